// msc_tcs.cuh -- tcgen05 block-diagonal inverse with E streamed from L2, for
// grids whose E does not fit in shared memory (n > 224; see msc_tc.cuh for the
// arithmetic, which is the same: BF16x3 products with FP32 accumulators, beta
// applied before the division by pkd + lam formed in FP64).
//
// Both products walk K in steps of 16.  The A operand of a step -- all kp rows
// of E^T or E against 16 columns, hi and lo parts, 2 x 32 kp bytes -- is one
// contiguous piece of an image laid out for it:
//   image 1 (E^T x):  [z / 8][k / 8][8 z][8 k]   MN-major A (M = k, K = z)
//   image 2 (E y):    [k / 8][z / 8][8 z][8 k]   K-major A  (M = z, K = k)
// In both, the stride between 8-blocks of M is 128 bytes and between 8-blocks
// of K kp / 8 x 128.  One thread copies the pieces with cp.async.bulk into a
// ring of S stages (full barriers count bytes, empty barriers are tcgen05
// commits), S - 1 steps ahead of the MMAs and across the two products and the
// tiles, since the sequence of pieces is always the same.
//
// A tile is N / 2 channels (N columns: re, im).  Its B operand (x, then y, hi
// and lo: 4 N kp bytes) stays in shared memory; the accumulators of the second
// product overwrite those of the first (mt N <= 512 TMEM columns).  What
// bounds it: E from L2, 128 kp^2 / N bytes per channel and product pair (n = 300,
// N = 128: 11.6 KB a channel against 4.8 KB of x and u in HBM) and the phases
// of a tile that follow one another (stage, product, sums, y, product, store).
// While thread 0 feeds the ring, the other lanes of its warp wait at a warp barrier
// and one lane of every other warp polls for the end of the product: with all 512
// threads polling, thread 0 got to run half as often (a product took 50000 cycles
// instead of 25000; 12800 are the MMAs).
// Measured, 26244 rows x 300: 159 us (N = 128), 252 us (N = 64), before the single
// polls 226 and 384, CUDA cores 880 us.
// It runs only where the caller sets tensor_cores=True.  BF16x3 is 13 times as far from
// 64 bits as the CUDA cores' FP32 products (6.1e-6 against 4.6e-7 at n = 300, 2-norm), and
// although the FP64 residual decides when a solve ends (|u - A psi| <= rtol |u|), the
// stiff components of the last correction keep the inverse's error: left to the
// autotuner, psi of the 81 x 81 x 300 batch was up to 4.6 times as far off.
#pragma once

#include "msc_tc.cuh"

namespace msc {
namespace tc {

constexpr int kStreamMaxK = 560;        // two stages and 32 channels fit in 227 KB up to here

// Dynamic shared memory: ring, B hi and lo, tables.
__host__ __device__ constexpr size_t stream_stage_bytes(int kp) { return (size_t)64 * kp; }
__host__ __device__ constexpr size_t stream_smem(int kp, int N, int S)
{
    return S * stream_stage_bytes(kp) + (size_t)4 * N * kp + 1024;
}

// The two images: one contiguous piece [hi, lo][2 K blocks][kp / 8][8 z][8 k] per 16
// of K, K = z in zk (E^T x) and K = k in kz (E y); zero past n.
__global__ void k_stream_images(int n, int kp, const double *__restrict__ E, __nv_bfloat16 *__restrict__ zk,
                                __nv_bfloat16 *__restrict__ kz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kp * kp) return;
    const int z = i / kp, k = i - z * kp, kb = kp / 8;
    const double v = z < n && k < n ? E[(size_t)z * n + k] : 0.0;
    const __nv_bfloat16 hi = __float2bfloat16_rn((float)v);
    const __nv_bfloat16 lo = __float2bfloat16_rn((float)(v - (double)__bfloat162float(hi)));
    const size_t part = (size_t)16 * kp, in = (size_t)(z % 8) * 8 + k % 8;
    const size_t a = (size_t)(z / 16) * 2 * part + ((size_t)(z / 8 % 2) * kb + k / 8) * 64 + in;
    const size_t b = (size_t)(k / 16) * 2 * part + ((size_t)(k / 8 % 2) * kb + z / 8) * 64 + in;
    zk[a] = hi;
    zk[a + part] = lo;
    kz[b] = hi;
    kz[b + part] = lo;
}

struct TcStreamParams {
    TcParams t;                          // e_img unused
    const __nv_bfloat16 *img1, *img2;    // [piece][hi, lo][2 K blocks][kp / 8][8][8]
};

// mbar_wait by one lane for its warp: sixteen polls instead of 512.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, int lane)
{
    bool done = true;
    if (lane == 0) done = mbar_wait(bar, parity);
    return __shfl_sync(0xffffffffu, done, 0);
}

template <int N, int S>
__global__ void __launch_bounds__(kThreads, 1) k_block_inverse_tcs(TcStreamParams sp)
{
    static_assert(N == 128 || N == 64, "a column group is 32 or 16 columns wide");
    const TcParams &prm = sp.t;
    constexpr int TR = N / 2;                 // channels per tile
    constexpr int CW = N / 4;                 // columns per warp (4 column groups)
    constexpr int NCH = CW / 16;              // 16-column chunks per warp
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[S], empty[S], bar_mma;
    __shared__ uint32_t tmem_base_s;
    __shared__ float sm_part[4][N];           // Sherman-Morrison partial sums per lane quarter
    __shared__ float2 beta_s[TR];
    __shared__ double pkd_s[TR];
    __shared__ double lam_s[kStreamMaxK];
    __shared__ float en_s[kStreamMaxK];
    __shared__ int next_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lq = warp & 3, c_begin = (warp >> 2) * CW;
    const int n = prm.n, kp = prm.kp, mt_count = prm.mt;
    const int kb = kp >> 3, ksteps = kp >> 4;
    const uint32_t half = (uint32_t)32 * kp;              // hi (or lo) part of a piece
    unsigned char *b_hi = smem + S * stream_stage_bytes(kp);
    unsigned char *b_lo = b_hi + (size_t)N * kp * 2;
    const uint32_t ring_a = smem_u32(smem), b_hi_a = smem_u32(b_hi), b_lo_a = smem_u32(b_lo);
    const uint32_t b_lbo = (uint32_t)N * 16u;             // B: stride between K blocks
    const uint32_t a_lbo = (uint32_t)kb * 128u;           // A: stride between K blocks
    uint32_t ncols = 32;
    while (ncols < (uint32_t)(mt_count * N)) ncols <<= 1;

    if (warp == 0) tmem_alloc(&tmem_base_s, ncols);
    for (int k = tid; k < kp; k += kThreads) {
        lam_s[k] = k < n ? prm.lam[k] : 0.0;
        en_s[k] = k < n ? (float)prm.en[k] : 0.f;
    }
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&bar_mma, 1);
        mbar_fence_init();
    }
    auto find_active = [&](int t) {
        for (; t < prm.ntiles; t += gridDim.x) {
            if (!prm.gate) return t;
            const int r0 = t * TR, nr = min(TR, prm.rows - r0);
            const int s0 = prm.row_sys[r0], s1 = prm.row_sys[r0 + nr - 1];
            for (int q = s0; q <= s1; ++q)
                if (prm.gate[q]) return t;
        }
        return prm.ntiles;
    };
    if (tid == 0) next_s = find_active(blockIdx.x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    int tile = next_s;
    __syncthreads();            // every thread has read next_s before the loop rewrites it
    bool ok = true;

    // thread 0: pieces consumed (MMAs issued) and copies issued, counted over
    // the whole life of the CTA; piece j sits in stage j % S
    int used = 0, issued = 0;
    auto issue = [&]() {
        const int ph = issued % (2 * ksteps), st = issued % S;
        const __nv_bfloat16 *src = ph < ksteps ? sp.img1 + (size_t)ph * 32 * kp
                                               : sp.img2 + (size_t)(ph - ksteps) * 32 * kp;
        mbar_expect_tx(&full[st], 2u * half);
        bulk_g2s(smem + (size_t)st * stream_stage_bytes(kp), src, 2u * half, &full[st]);
        ++issued;
    };
    if (tid == 0 && tile < prm.ntiles)
        for (int s = 0; s < S; ++s) issue();

    // One product (thread 0): D[m] (+)= A_hi B_hi + A_hi B_lo + A_lo B_hi over the
    // ksteps pieces; `last`: no copy past the end of this product
    auto run_product = [&](uint32_t idesc, bool last) {
        const int end = used + ksteps;
        for (int s = 0; s < ksteps; ++s) {
            const int st = used % S;
            if (!mbar_wait(&full[st], (uint32_t)(used / S) & 1u)) return false;
            const uint32_t a = ring_a + (uint32_t)st * (uint32_t)stream_stage_bytes(kp);
            const uint32_t b_off = (uint32_t)(2 * s) * b_lbo;
            const uint64_t bh = make_desc(b_hi_a + b_off, b_lbo, 128);
            const uint64_t bl = make_desc(b_lo_a + b_off, b_lbo, 128);
            for (int m = 0; m < mt_count; ++m) {
                const uint32_t d = tmem + (uint32_t)(m * N);
                const uint64_t ah = make_desc(a + (uint32_t)m * 2048u, a_lbo, 128);
                const uint64_t al = make_desc(a + half + (uint32_t)m * 2048u, a_lbo, 128);
                mma_bf16(d, ah, bh, idesc, s > 0 ? 1u : 0u);
                mma_bf16(d, ah, bl, idesc, 1u);
                mma_bf16(d, al, bh, idesc, 1u);
            }
            mma_commit(&empty[st]);
            ++used;
            // refill the stage of the previous piece once its MMAs are done
            // (this piece's MMAs are queued meanwhile)
            if (used >= 2 && issued < used - 1 + S && (!last || issued < end)) {
                const int pv = used - 2;
                if (!mbar_wait(&empty[pv % S], (uint32_t)(pv / S) & 1u)) return false;
                issue();
            }
        }
        return true;
    };
    const uint32_t idesc_mn = make_idesc(N, 1, 0);   // E^T x: A MN-major, B K-major
    const uint32_t idesc_k = make_idesc(N, 0, 1);    // E y:   A K-major, B MN-major
    uint32_t mma_phase = 0;

    while (tile < prm.ntiles && ok) {
        const int row0 = tile * TR;
        const int nrow = min(TR, prm.rows - row0);
        for (int j = tid; j < TR; j += kThreads) pkd_s[j] = j < nrow ? prm.row_pkd[row0 + j] : 0.0;
        // ---- stage x: a thread takes 8 consecutive z of one channel (64 bytes)
        // and writes its four 16-byte units (re, im x hi, lo).  Lanes: 8
        // channels x 4 z-blocks (256 contiguous bytes of each row; the stores of
        // 8 channels of one z-block cover all banks twice).
        constexpr int kCG = TR / 8;                       // channel groups of 8
        const int units = kCG * ((kb + 3) / 4);           // of 8 channels x 4 z-blocks
        const bool vec = (n % 2 == 0) && (reinterpret_cast<uintptr_t>(prm.x) & 15u) == 0;
        for (int u = warp; u < units; u += kThreads / 32) {
            const int j = (u % kCG) * 8 + (lane & 7), zb = (u / kCG) * 4 + (lane >> 3);
            if (zb >= kb) continue;
            float2 v[8];
            const float2 *xr = prm.x + (size_t)(row0 + j) * n + zb * 8;
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const int z = zb * 8 + e;
                if (vec) {
                    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (j < nrow && z < n) t = *reinterpret_cast<const float4 *>(xr + e);
                    v[e] = make_float2(t.x, t.y);
                    v[e + 1] = make_float2(t.z, t.w);
                } else {
                    v[e] = (j < nrow && z < n) ? xr[e] : make_float2(0.f, 0.f);
                    v[e + 1] = (j < nrow && z + 1 < n) ? xr[e + 1] : make_float2(0.f, 0.f);
                }
            }
            uint32_t rh[4], ih[4], rl[4], il[4];
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const __nv_bfloat162 hr = __floats2bfloat162_rn(v[e].x, v[e + 1].x);
                const __nv_bfloat162 hi = __floats2bfloat162_rn(v[e].y, v[e + 1].y);
                const float2 fr = __bfloat1622float2(hr), fi = __bfloat1622float2(hi);
                const __nv_bfloat162 lr = __floats2bfloat162_rn(v[e].x - fr.x, v[e + 1].x - fr.y);
                const __nv_bfloat162 li = __floats2bfloat162_rn(v[e].y - fi.x, v[e + 1].y - fi.y);
                rh[e >> 1] = *reinterpret_cast<const uint32_t *>(&hr);
                ih[e >> 1] = *reinterpret_cast<const uint32_t *>(&hi);
                rl[e >> 1] = *reinterpret_cast<const uint32_t *>(&lr);
                il[e >> 1] = *reinterpret_cast<const uint32_t *>(&li);
            }
            const uint32_t o_re = kmaj_off(2 * j, zb * 8, N), o_im = o_re + 16;
            *reinterpret_cast<uint4 *>(b_hi + o_re) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
            *reinterpret_cast<uint4 *>(b_hi + o_im) = make_uint4(ih[0], ih[1], ih[2], ih[3]);
            *reinterpret_cast<uint4 *>(b_lo + o_re) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
            *reinterpret_cast<uint4 *>(b_lo + o_im) = make_uint4(il[0], il[1], il[2], il[3]);
        }
        fence_proxy_async();
        __syncthreads();

        // ---- E^T x
        if (tid == 0) {
            tc_fence_after();
            ok = run_product(idesc_mn, false);
            mma_commit(&bar_mma);
        }
        __syncwarp();           // lanes that polled bar_mma meanwhile would hold thread 0 up
        // the next active tile, while the MMAs run (every thread read next_s
        // before the previous tile's last barrier); its rows go to L2
        if (tid == 32) {
            const int nx = find_active(tile + gridDim.x);
            next_s = nx;
            if (nx < prm.ntiles) {
                const int r0 = nx * TR;
                const uint32_t bytes = (uint32_t)min(TR, prm.rows - r0) * (uint32_t)n * 8u;
                const float2 *src = prm.x + (size_t)r0 * n;
                if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes & ~15u)
                                 : "memory");
            }
        }
        if (!mbar_wait_warp(&bar_mma, mma_phase, lane)) ok = false;
        mma_phase ^= 1u;
        tc_fence_after();
        if (!__syncthreads_and(ok)) { ok = false; break; }

        // ---- s_j = sum_k en_k xt_kj / (pkd_j + lam_k): a thread adds its k of every
        // M tile, then the lanes (butterfly) and the lane quarters in FP64, in a
        // fixed order
        {
            float acc[NCH][16];
#pragma unroll
            for (int q = 0; q < NCH; ++q)
#pragma unroll
                for (int c = 0; c < 16; ++c) acc[q][c] = 0.f;
            for (int m = 0; m < mt_count; ++m) {
                const int k0 = m * 128 + lq * 32;
                if (k0 >= n) break;                        // warp-uniform
                const int k = k0 + lane;
                float vv[kLdChunks][16];
                tmem_ld_chunks(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(m * N + c_begin), NCH, vv);
                if (k < n) {
                    const double lam_k = lam_s[k];
                    const float en_k = en_s[k];
#pragma unroll
                    for (int q = 0; q < NCH; ++q)
#pragma unroll
                        for (int c = 0; c < 16; c += 2) {
                            const float w = en_k * shifted_inverse(pkd_s[(c_begin + 16 * q + c) >> 1], lam_k);
                            acc[q][c] = fmaf(w, vv[q][c], acc[q][c]);
                            acc[q][c + 1] = fmaf(w, vv[q][c + 1], acc[q][c + 1]);
                        }
                }
            }
#pragma unroll
            for (int q = 0; q < NCH; ++q) {
                const float sum = warp_reduce_scatter16(acc[q], lane);
                if ((lane & 1) == 0) sm_part[lq][c_begin + 16 * q + ((lane >> 1) & 15)] = sum;
            }
        }
        __syncthreads();
        for (int j = tid; j < TR; j += kThreads) {
            double sr = 0.0, si = 0.0;
            for (int w = 0; w < 4; ++w) {
                sr += sm_part[w][2 * j];
                si += sm_part[w][2 * j + 1];
            }
            const double2 b = j < nrow ? cmul(prm.row_cf[row0 + j], make_double2(sr, si))
                                       : make_double2(0.0, 0.0);
            beta_s[j] = make_float2((float)b.x, (float)b.y);
        }
        __syncthreads();

        // ---- y = (xt + beta en) / (pkd + lam) as the MN-major B operand of E y (rows
        // k in [n, kp) are zero)
        for (int m = 0; m < mt_count; ++m) {
            const int k0 = m * 128 + lq * 32;
            if (k0 >= kp) break;                           // warp-uniform
            const int k = k0 + lane;
            float vv[kLdChunks][16];
            tmem_ld_chunks(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(m * N + c_begin), NCH, vv);
            if (k >= kp) continue;
            const bool valid = k < n;
            const double lam_k = lam_s[k];
            const float en_k = en_s[k];
#pragma unroll
            for (int q = 0; q < NCH; ++q) {
                const int c0 = c_begin + 16 * q;
                uint32_t hw[8], lw[8];
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    const int j = (c0 + c) >> 1;
                    float yr = 0.f, yi = 0.f;
                    if (valid && j < nrow) {
                        const float inv = shifted_inverse(pkd_s[j], lam_k);
                        const float2 b = beta_s[j];
                        yr = (vv[q][c] + b.x * en_k) * inv;
                        yi = (vv[q][c + 1] + b.y * en_k) * inv;
                    }
                    const __nv_bfloat162 h = __floats2bfloat162_rn(yr, yi);
                    const float2 fh = __bfloat1622float2(h);
                    const __nv_bfloat162 l = __floats2bfloat162_rn(yr - fh.x, yi - fh.y);
                    hw[c >> 1] = *reinterpret_cast<const uint32_t *>(&h);
                    lw[c >> 1] = *reinterpret_cast<const uint32_t *>(&l);
                }
                const uint32_t o = (uint32_t)(((k >> 3) * (N >> 3) + (c0 >> 3)) * 128 + (k & 7) * 16);
                *reinterpret_cast<uint4 *>(b_hi + o) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                *reinterpret_cast<uint4 *>(b_hi + o + 128) = make_uint4(hw[4], hw[5], hw[6], hw[7]);
                *reinterpret_cast<uint4 *>(b_lo + o) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                *reinterpret_cast<uint4 *>(b_lo + o + 128) = make_uint4(lw[4], lw[5], lw[6], lw[7]);
            }
        }
        tc_fence_before();
        fence_proxy_async();
        __syncthreads();

        // ---- E y over the same accumulator columns
        const int next = next_s;
        if (tid == 0) {
            tc_fence_after();
            ok = run_product(idesc_k, next >= prm.ntiles);
            mma_commit(&bar_mma);
        }
        __syncwarp();
        if (!mbar_wait_warp(&bar_mma, mma_phase, lane)) ok = false;
        mma_phase ^= 1u;
        tc_fence_after();
        if (!__syncthreads_and(ok)) { ok = false; break; }

        // ---- u rows (z contiguous across lanes)
        for (int m = 0; m < mt_count; ++m) {
            const int z0 = m * 128 + lq * 32;
            if (z0 >= n) break;                            // warp-uniform
            const int z = z0 + lane;
            float vv[kLdChunks][16];
            tmem_ld_chunks(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(m * N + c_begin), NCH, vv);
            if (z >= n) continue;
#pragma unroll
            for (int q = 0; q < NCH; ++q)
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    const int j = (c_begin + 16 * q + c) >> 1;
                    if (j < nrow)
                        prm.out[(size_t)(row0 + j) * n + z] = make_float2(vv[q][c], vv[q][c + 1]);
                }
        }
        tc_fence_before();
        __syncthreads();
        tile = next;
    }

    if (!ok && tid == 0 && prm.error) atomicExch(prm.error, 1);
    // nothing may land or run after the kernel leaves: copies in flight, and
    // (after a time-out) the MMAs the last commit covers
    if (tid == 0) {
        for (int j = used; j < issued; ++j) (void)mbar_wait(&full[j % S], (uint32_t)(j / S) & 1u);
        if (!ok) (void)mbar_wait(&bar_mma, mma_phase ^ 1u);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem_base_s, ncols);
}

}  // namespace tc
}  // namespace msc
