// msc_dmma.cuh -- FP64 tensor-core (DMMA) forms of the block-diagonal inverse
// and of the residual's diagonal part.
//
// Both are products of an n x n operator matrix (E^T, E or T) with the 2 C
// real columns of C channel rows:  M = n, K = n, N = 2 channels.  tcgen05 has
// no FP64 kind, so the FP64 tensor path of sm_100a is mma.sync m8n8k4.f64; it
// runs at the FP64 pipe's rate (measured 36.9 TFLOP/s against 32.4 for plain
// DFMA loops) but takes one operand register per 256 multiply-adds instead of
// one per few, which is what bounded the CUDA-core kernels these replace
// (shared-memory and L2 operand loads, about a third of the FP64 peak).
//
// Operand layouts.
//   A: a "fragment image" of the matrix, [m-tile of 8][k-step of 8][lane] of
//      double2: lane l holds A(8 mt + l/4, 8 ks + 2 (l%4) + {0, 1}).  A warp's
//      operand of one k-step is one coalesced 512-byte load; rows and columns
//      past n are zero, so no load needs a bounds test.
//   B: shared memory [column][LDZ], z contiguous: lane l reads the pair
//      (8 ks + 2 (l%4) + {0, 1}) of column 8 j + l/4 as one 16-byte load.  LDZ
//      is 8 mod 16 doubles, which spreads a quarter-warp over all banks.
//   The pair order inside a k-step is the same for A and B, so the sum over K
//   is complete; even columns are the real parts, odd ones the imaginary
//   parts of a channel, and an accumulator pair (c0, c1) is one complex value.
//
// Work split.  A CTA of 8 warps (4 along M x 2 along N) owns 8 NTW channels
// (16 NTW columns); a cluster of CL CTAs shares one channel tile, the m-tiles of
// both products dealt out evenly over its 4 CL warp rows (MT or MT - 1 each).
// The cluster exchanges the Sherman-Morrison partial sums and the scaled
// coefficients through distributed shared memory.  CL > 1 is what keeps the
// GPU busy on one beam (a 100-channel system is 13 tiles for 148 SMs) and what
// lets n up to 1024 keep its accumulators in registers.
#pragma once

#include <cooperative_groups.h>

#include "msc_common.cuh"

namespace msc {
namespace dm {

constexpr int kThreads = 256;
constexpr int kWM = 4, kWN = 2;          // warps along M and along N

__device__ __forceinline__ void mma_f64(double2 &c, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c.x), "+d"(c.y)
        : "d"(a), "d"(b));
}

__host__ __device__ constexpr int ksteps(int n) { return (n + 7) / 8; }
// doubles between two columns of the B buffer: >= 8 ksteps, 8 mod 16
__host__ __device__ constexpr int col_stride(int n) { return ksteps(n) * 8 + (ksteps(n) % 2 ? 0 : 8); }
__host__ __device__ constexpr size_t image_elems(int n) { return (size_t)ksteps(n) * ksteps(n) * 32; }

// Fragment image of A(m, k) = src[m * n + k] (transpose = 0) or src[k * n + m].
__global__ void k_fragment_image(int n, const double *__restrict__ src, int transpose,
                                 double2 *__restrict__ img)
{
    const int ks_n = ksteps(n);
    const size_t total = image_elems(n);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(i & 31);
        const int ks = (int)((i >> 5) % ks_n), mt = (int)((i >> 5) / ks_n);
        const int m = mt * 8 + (lane >> 2), k = ks * 8 + 2 * (lane & 3);
        double2 v = make_double2(0.0, 0.0);
        if (m < n && k < n) v.x = transpose ? src[(size_t)k * n + m] : src[(size_t)m * n + k];
        if (m < n && k + 1 < n) v.y = transpose ? src[(size_t)(k + 1) * n + m] : src[(size_t)m * n + k + 1];
        img[i] = v;
    }
}

// acc[i][j] (i < CNT <= MT) = m-tile i of the warp times its NTW column tiles.
// img: the image at the warp's first m-tile and lane.  U k-steps of A are in
// flight ahead of their use (L2 latency: few warps run on small systems); the
// loop body has no branch, so that the loads stay ahead of the products.
template <int CNT, int MT, int NTW, int U>
__device__ __forceinline__ void product_run(const double2 *__restrict__ img, size_t tile_stride, int ks_n,
                                            const double *bcol, int ldz, double2 (&acc)[MT][NTW])
{
    double2 a[U][CNT];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < CNT; ++i)
            a[u][i] = __ldg(img + i * tile_stride + (size_t)min(u, ks_n - 1) * 32);
    auto step = [&](int ks, double2 (&au)[CNT]) {
        double2 b[NTW];
#pragma unroll
        for (int j = 0; j < NTW; ++j)
            b[j] = *reinterpret_cast<const double2 *>(bcol + (size_t)j * 8 * ldz + ks * 8);
#pragma unroll
        for (int i = 0; i < CNT; ++i)
#pragma unroll
            for (int j = 0; j < NTW; ++j) mma_f64(acc[i][j], au[i].x, b[j].x);
#pragma unroll
        for (int i = 0; i < CNT; ++i)
#pragma unroll
            for (int j = 0; j < NTW; ++j) mma_f64(acc[i][j], au[i].y, b[j].y);
        const size_t nx = (size_t)min(ks + U, ks_n - 1) * 32;
#pragma unroll
        for (int i = 0; i < CNT; ++i) au[i] = __ldg(img + i * tile_stride + nx);
    };
    int k0 = 0;
    for (; k0 + U <= ks_n; k0 += U)
#pragma unroll
        for (int u = 0; u < U; ++u) step(k0 + u, a[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (k0 + u < ks_n) step(k0 + u, a[u]);
}

// mcount is MT or MT - 1 (an even deal of the m-tiles over the warps).
template <int MT, int NTW, int U>
__device__ __forceinline__ void product(const double2 *__restrict__ img, size_t tile_stride, int mcount,
                                        int ks_n, const double *bcol, int ldz, double2 (&acc)[MT][NTW])
{
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTW; ++j) acc[i][j] = make_double2(0.0, 0.0);
    if (mcount == MT)
        product_run<MT, MT, NTW, U>(img, tile_stride, ks_n, bcol, ldz, acc);
    else if constexpr (MT > 1)
        product_run<MT - 1, MT, NTW, U>(img, tile_stride, ks_n, bcol, ldz, acc);
}

struct Params {
    int n, rows;                   // nodes; channel rows in all
    const double2 *img1, *img2;    // E^T and E (block inverse); T and null (residual)
    const double *lam, *en;        // block inverse
    const double2 *row_cf;         // c / (1 - c f_n) per row (block inverse)
    const double *v00;             // residual
    const double2 *row_c, *row_rhs;
    const double *row_pkd;
    const int *row_sys, *gate;
    const double2 *x;
    double2 *out;
    int flag;                      // block inverse: out += ; residual: add the right-hand side
};

// Shared memory of a CTA: the column buffer, then per-row scalars and sums.
template <int NTW>
__host__ __device__ constexpr size_t smem_bytes(int n, int cl)
{
    const size_t cols = 16 * NTW, tr = 8 * NTW;
    return (cols * col_stride(n) + tr + 2 * tr * (kWM + cl + 1) + 2 * 32 * 8) * sizeof(double);
}

// The two halves of a cluster barrier; the arrival orders no memory, it only says that
// the CTA has started.
__device__ __forceinline__ void cluster_arrive()
{
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// Any system of rows [row0, row0 + nrow) still active?  (same answer in every thread)
__device__ __forceinline__ bool tile_active(const Params &p, int row0, int nrow)
{
    if (!p.gate) return true;
    const int s1 = __ldg(p.row_sys + row0 + nrow - 1);
    for (int s = __ldg(p.row_sys + row0); s <= s1; ++s)
        if (p.gate[s]) return true;
    return false;
}

// x rows -> columns [2 r] (re), [2 r + 1] (im) of the B buffer, zero past n
// and past nrow.
template <int NTW>
__device__ __forceinline__ void stage_rows(const Params &p, int row0, int nrow, double *Xs, int ldz)
{
    constexpr int TR = 8 * NTW;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kz = ksteps(p.n) * 8;
    for (int z0 = 0; z0 < kz; z0 += 32) {
        const int z = z0 + lane;
        double2 v[NTW];
#pragma unroll
        for (int q = 0; q < NTW; ++q) {
            const int r = warp + 8 * q;
            v[q] = make_double2(0.0, 0.0);
            if (r < nrow && z < p.n) v[q] = p.x[(size_t)(row0 + r) * p.n + z];
        }
        if (z < kz) {
#pragma unroll
            for (int q = 0; q < NTW; ++q) {
                const int r = warp + 8 * q;
                Xs[(size_t)(2 * r) * ldz + z] = v[q].x;
                Xs[(size_t)(2 * r + 1) * ldz + z] = v[q].y;
            }
        }
    }
    static_assert(TR == 8 * NTW, "one row of the tile per warp and pass");
}

// Block-diagonal inverse out (=|+=) D^-1 x (see k_block_inverse for the
// formulas): E^T x by DMMA, the Sherman-Morrison scalar and the division by
// pkd + lam on the accumulators in registers, E y by DMMA.
// Grid: channel tiles x CL, clusters of CL CTAs along x.
template <int MT, int NTW, int U>
__global__ void __launch_bounds__(kThreads, 2) k_block_inverse_dmma(Params p)
{
    namespace cg = cooperative_groups;
    constexpr int TR = 8 * NTW, NC = 2 * TR;
    extern __shared__ __align__(16) double dsm[];
    const cg::cluster_group cluster = cg::this_cluster();
    const int cl = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int ldz = col_stride(p.n), ks_n = ksteps(p.n);
    double *Xs = dsm;                                            // [NC][ldz]
    double *pkd_s = Xs + (size_t)NC * ldz;                       // [TR]
    double2 *sred = reinterpret_cast<double2 *>(pkd_s + TR);     // [kWM][TR]
    double2 *sall = sred + kWM * TR;                             // [cl][TR]
    double2 *beta_s = sall + (size_t)cl * TR;                    // [TR]
    const int row0 = (int)(blockIdx.x / cl) * TR;
    const int nrow = min(TR, p.rows - row0);
    if (!tile_active(p, row0, nrow)) return;                     // same for the whole cluster
    // Shared memory of another CTA may be touched once that CTA runs: the arrival is
    // waited for where the sums are sent, behind the first product.
    if (cl > 1) cluster_arrive();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp & (kWM - 1), wn = warp >> 2;
    const int g = lane >> 2, q = lane & 3;
    // m-tiles of this warp: mt0, mt0 + ms, ... (MT or MT - 1 of them)
    const int mt0 = rank * kWM + wm, ms = cl * kWM;
    const int mcount = mt0 < ks_n ? (ks_n - 1 - mt0) / ms + 1 : 0;
    const size_t tstride = (size_t)ms * ks_n * 32;
    const size_t ioff = ((size_t)mt0 * ks_n) * 32 + lane;
    const double *bcol = Xs + (size_t)(wn * NTW * 8 + g) * ldz + 2 * q;

    stage_rows<NTW>(p, row0, nrow, Xs, ldz);
    for (int r = threadIdx.x; r < TR; r += kThreads) pkd_s[r] = r < nrow ? p.row_pkd[row0 + r] : 0.0;
    __syncthreads();

    double2 acc[MT][NTW];
    product<MT, NTW, U>(p.img1 + ioff, tstride, mcount, ks_n, bcol, ldz, acc);

    // s_r = sum_k en_k xt_kr / (pkd_r + lam_k) over this CTA's k: thread, then
    // the 8 lanes of a column, then warps, then CTAs, in a fixed order
    double2 s[NTW];
#pragma unroll
    for (int j = 0; j < NTW; ++j) s[j] = make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int k = (mt0 + i * ms) * 8 + g;
        if (i >= mcount || k >= p.n) break;
        const double lk = __ldg(p.lam + k), ek = __ldg(p.en + k);
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
            const int r = (wn * NTW + j) * 4 + q;
            const double w = ek / (pkd_s[r] + lk);
            if (r < nrow) {
                s[j].x = fma(w, acc[i][j].x, s[j].x);
                s[j].y = fma(w, acc[i][j].y, s[j].y);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            s[j].x += __shfl_xor_sync(0xffffffffu, s[j].x, o);
            s[j].y += __shfl_xor_sync(0xffffffffu, s[j].y, o);
        }
        if (g == 0) sred[wm * TR + (wn * NTW + j) * 4 + q] = s[j];
    }
    __syncthreads();
    if (cl > 1) {
        cluster_wait();        // every CTA of the cluster has started
        for (int t = threadIdx.x; t < cl * TR; t += kThreads) {
            const int dst = t / TR, r = t - dst * TR;
            double2 v = sred[r];
            for (int w = 1; w < kWM; ++w) v = cadd(v, sred[w * TR + r]);
            cluster.map_shared_rank(sall, dst)[rank * TR + r] = v;
        }
        cluster.sync();        // sums in place, and every CTA is done reading x
        for (int r = threadIdx.x; r < TR; r += kThreads) {
            double2 v = sall[r];
            for (int c = 1; c < cl; ++c) v = cadd(v, sall[c * TR + r]);
            beta_s[r] = r < nrow ? cmul(p.row_cf[row0 + r], v) : make_double2(0.0, 0.0);
        }
    } else {
        for (int r = threadIdx.x; r < TR; r += kThreads) {
            double2 v = sred[r];
            for (int w = 1; w < kWM; ++w) v = cadd(v, sred[w * TR + r]);
            beta_s[r] = r < nrow ? cmul(p.row_cf[row0 + r], v) : make_double2(0.0, 0.0);
        }
    }
    __syncthreads();

    // yt over x in the column buffers of all CTAs of the cluster (the zero rows
    // k in [n, 8 ksteps) stay)
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        const int k = (mt0 + i * ms) * 8 + g;
        if (i >= mcount || k >= p.n) break;
        const double lk = __ldg(p.lam + k), ek = __ldg(p.en + k);
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
            const int r = (wn * NTW + j) * 4 + q;
            double2 y = make_double2(0.0, 0.0);
            if (r < nrow) {
                const double inv = 1.0 / (pkd_s[r] + lk);
                const double2 b = beta_s[r];
                y = make_double2((acc[i][j].x + b.x * ek) * inv, (acc[i][j].y + b.y * ek) * inv);
            }
            const size_t o = (size_t)(2 * r) * ldz + k;
            if (cl > 1) {
                for (int c = 0; c < cl; ++c) {
                    double *d = cluster.map_shared_rank(Xs, c) + o;
                    d[0] = y.x;
                    d[ldz] = y.y;
                }
            } else {
                Xs[o] = y.x;
                Xs[o + ldz] = y.y;
            }
        }
    }
    if (cl > 1)
        cluster.sync();        // no remote access after this: CTAs may leave on their own
    else
        __syncthreads();

    product<MT, NTW, U>(p.img2 + ioff, tstride, mcount, ks_n, bcol, ldz, acc);
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
        const int r = (wn * NTW + j) * 4 + q;
        if (r >= nrow || (p.gate && p.gate[__ldg(p.row_sys + row0 + r)] == 0)) continue;
        double2 *o = p.out + (size_t)(row0 + r) * p.n;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int z = (mt0 + i * ms) * 8 + g;
            if (i >= mcount || z >= p.n) break;
            double2 v = acc[i][j];
            if (p.flag) v = cadd(v, o[z]);
            o[z] = v;
        }
    }
}

// Residual diagonal part out = b - D x (see k_residual_diag): T x by DMMA.
// Grid: (channel tiles, M slices); x is staged by every slice.
template <int MT, int NTW, int U>
__global__ void __launch_bounds__(kThreads, 2) k_residual_dmma(Params p)
{
    constexpr int TR = 8 * NTW;
    extern __shared__ __align__(16) double dsm[];
    const int ldz = col_stride(p.n), ks_n = ksteps(p.n);
    double *Xs = dsm;
    const int row0 = (int)blockIdx.x * TR;
    const int nrow = min(TR, p.rows - row0);
    if (!tile_active(p, row0, nrow)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp & (kWM - 1), wn = warp >> 2;
    const int g = lane >> 2, q = lane & 3;
    const int mt0 = (int)blockIdx.y * kWM + wm, ms = (int)gridDim.y * kWM;
    const int mcount = mt0 < ks_n ? (ks_n - 1 - mt0) / ms + 1 : 0;
    stage_rows<NTW>(p, row0, nrow, Xs, ldz);
    __syncthreads();
    double2 acc[MT][NTW];
    product<MT, NTW, U>(p.img1 + ((size_t)mt0 * ks_n) * 32 + lane, (size_t)ms * ks_n * 32, mcount, ks_n,
                        Xs + (size_t)(wn * NTW * 8 + g) * ldz + 2 * q, ldz, acc);
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
        const int r = (wn * NTW + j) * 4 + q;
        if (r >= nrow) continue;
        const int row = row0 + r;
        if (p.gate && p.gate[__ldg(p.row_sys + row)] == 0) continue;
        const double pk = p.row_pkd[row];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int z = (mt0 + i * ms) * 8 + g;
            if (i >= mcount || z >= p.n) break;
            const double diag = __ldg(p.v00 + z) + pk;
            const double2 xz = make_double2(Xs[(size_t)(2 * r) * ldz + z], Xs[(size_t)(2 * r + 1) * ldz + z]);
            double2 d = make_double2(acc[i][j].x + diag * xz.x, acc[i][j].y + diag * xz.y);
            if (z == p.n - 1) d = csub(d, cmul(p.row_c[row], xz));
            double2 o = make_double2(-d.x, -d.y);
            if (p.flag && z == p.n - 1) o = cadd(o, p.row_rhs[row]);
            p.out[(size_t)row * p.n + z] = o;
        }
    }
}

// ---- launch configuration ---------------------------------------------------
struct Config {
    int ntw, cl, mt;       // channels 8 ntw per CTA, M split cl, m-tiles per warp (template bound)
};

inline size_t smem_for(int ntw, int n, int cl)
{
    switch (ntw) {
    case 1: return smem_bytes<1>(n, cl);
    case 2: return smem_bytes<2>(n, cl);
    default: return smem_bytes<3>(n, cl);
    }
}

constexpr int kMaxSmem = 227 * 1024;

// m-tiles per warp of an M split over cl CTAs (instances: 1..5, with 1..3
// column tiles per warp).
inline int mt_of(int n, int cl) { return (ksteps(n) + kWM * cl - 1) / (kWM * cl); }
// Two CTAs per SM (128 registers): the accumulators take 4 MT NTW, the rest
// goes to A operands in flight (4 MT per k-step).
template <int MT, int NTW> struct Tune {
    static constexpr int room = (100 - 4 * MT * NTW - 4 * NTW) / (4 * MT);
    static constexpr int u = room < 1 ? 1 : room > 6 ? 6 : room;
};

// One (MT, NTW) instance of either kernel: its launch, or (launch = false) its
// shared-memory limit.
template <int MT, int NTW>
cudaError_t instance(bool inverse, const Config &c, const Params &p, cudaStream_t st, bool launch)
{
    using T = Tune<MT, NTW>;
    auto *inv = &k_block_inverse_dmma<MT, NTW, T::u>;
    auto *res = &k_residual_dmma<MT, NTW, T::u>;
    if (!launch) {
        cudaError_t e = cudaFuncSetAttribute(inv, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
        return e != cudaSuccess
                   ? e
                   : cudaFuncSetAttribute(res, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    }
    const int tiles = (p.rows + 8 * NTW - 1) / (8 * NTW);
    if (!inverse) {
        res<<<dim3(tiles, c.cl), kThreads, smem_for(NTW, p.n, 1), st>>>(p);
        return cudaPeekAtLastError();       // (the caller's own check still sees it)
    }
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(tiles * c.cl);
    lc.blockDim = dim3(kThreads);
    lc.dynamicSmemBytes = smem_for(NTW, p.n, c.cl);
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c.cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, inv, p);
}

inline cudaError_t dispatch(bool inverse, const Config &c, const Params &p, cudaStream_t st, bool launch)
{
#define MSC_DM_CASE(MT, NTW) \
    if (c.mt == MT && c.ntw == NTW) return instance<MT, NTW>(inverse, c, p, st, launch);
    MSC_DM_CASE(1, 1) MSC_DM_CASE(1, 2) MSC_DM_CASE(1, 3)
    MSC_DM_CASE(2, 1) MSC_DM_CASE(2, 2) MSC_DM_CASE(2, 3)
    MSC_DM_CASE(3, 1) MSC_DM_CASE(3, 2) MSC_DM_CASE(3, 3)
    MSC_DM_CASE(4, 1) MSC_DM_CASE(4, 2) MSC_DM_CASE(4, 3)
    MSC_DM_CASE(5, 1) MSC_DM_CASE(5, 2) MSC_DM_CASE(5, 3)
#undef MSC_DM_CASE
    return cudaErrorInvalidValue;
}

inline cudaError_t set_attributes()
{
    for (int mt = 1; mt <= 5; ++mt)
        for (int ntw = 1; ntw <= 3; ++ntw) {
            cudaError_t e = dispatch(true, Config{ntw, 1, mt}, Params{}, nullptr, false);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// Split of R rows (measured on B200, us of the block inverse, both products; before: the CUDA-core kernel):
//   rows x n        ntw/cl and us                                      before
//   121 x 100       1/1 12.9   1/2 12.9   1/4 8.8    1/8 10.9            33
//   100 x 550       1/4 46     1/8 31     2/8 48                        635
//   1681 x 200      1/2 40     2/2 40     3/2 40     3/4 37             118
//   26244 x 300     1/2 812    2/2 747    3/2 896 (one CTA per SM)     2854
//   119409 x 150    1/1 977    2/1 851    3/1 784    3/2 1080          2681
// So: the smallest cluster whose warps hold at most 5 m-tiles; wide tiles
// (less A traffic per product) once they give every SM work, as wide as two
// CTAs' column buffers fit in one SM; and for few rows narrow tiles with the
// M rows split further while every CTA still has an SM to itself and more
// than one m-tile per warp.  784 us is 74% of the DMMA rate.
// The residual (one product, x staged by every M slice) takes the same split; measured,
// us at it / at its own best: 121 x 100 5.1 / 5.1, 100 x 550 17.0 / 17.0, 1681 x 200 21.1 /
// 19.5 (3/4), 26244 x 300 386 / 386, 29856 x 150 140 / 137 (2/1), 119409 x 150 461 / 461.
inline Config choose(int rows, int n, int sms)
{
    int cl = 1;
    while (mt_of(n, cl) > 5) cl *= 2;
    const int narrow = (rows + 7) / 8;
    if (narrow * cl <= 2 * sms) {
        while (cl < 8 && 2 * cl * narrow <= sms && mt_of(n, cl) > 1) cl *= 2;
        return Config{1, cl, mt_of(n, cl)};
    }
    const int ntw = 2 * (smem_for(3, n, cl) + 1024) <= 228 * 1024 ? 3
                  : 2 * (smem_for(2, n, cl) + 1024) <= 228 * 1024 ? 2 : 1;
    return Config{ntw, cl, mt_of(n, cl)};
}

}  // namespace dm
}  // namespace msc
