// msc_halo.cuh -- channel coupling over halo tiles, for tap windows that do not
// factorise (and the masked couplings of the Gauss-Seidel form):
//   out[r] = in0[r] + sgn sum_t V_t(z) src[pos(r) - delta_t](z),   sgn = +-1
//
// A block owns a patch of bx x by torus positions (at most 8 x 8) of one system and
// the ZC z of one 128-byte line.  It stages the taps of the window and the patch with
// a halo of HX, HY positions, the reach of the taps, in shared memory; absent channels
// (outside a truncated set) read as zero and positions wrap around the torus as the
// reference's modulo(G_j - G_i, n).  A thread keeps one column of YS + 2 HY halo values
// in registers and produces YS outputs along y for one (x, z): a value loaded once
// serves up to 2 HY + 1 taps.  NS threads share a patch column (by <= NS YS).
//
// What bounds it: the (2 HX + 1)(2 HY + 1) complex FMAs per element (41 x 41 x 200
// with 81 taps: 3.0 us in FP32, 5.9 us in FP64) on large systems, and below that the
// launch and the chain of dependent loads before the first of them (about 4.5 us).  So:
//  - patches divide the torus evenly (41 = 6 x 7 instead of 6 x 8: 1.05 instead of 1.37
//    times the outputs) and a block takes one line of z, half of what it took before;
//  - a patch is two segments of by <= 8 high where that still gives three blocks per
//    SM: it reads 3.4 instead of 4.6 values per output and computes the rows of fewer
//    halo positions (FP32 13.0 -> 11.4 us, FP64 20.4 -> 18.7 us at 41 x 41 x 200);
//    smaller systems keep one segment, which gives them more blocks;
//  - taps and halo come by cp.async, all of a thread's copies in flight at once (a loop
//    of tap index, tap, store took a round trip to L2 per step), and the outputs' in0
//    is fetched behind them;
//  - FP32 sums with packed FMAs (see BoxMac).
// Measured, us per launch, before -> now: 41 x 41 x 200 FP32 14.6 -> 11.4, FP64 22.8 ->
// 18.7; 9 x 9 x 91 FP64 7.8 -> 6.0; 7 x 5 x 81 with 25 taps 5.4 -> 5.0.
#pragma once

#include "msc_box.cuh"

namespace msc {

struct CouplingTiles {
    const int4 *work;         // [nwork]: system, x0, y0
    const int *pos_row;       // [B][nkx * nky]: row of each torus position, -1 if absent
    const int *tap_window;    // [(2 HX + 1) * (2 HY + 1)]: tap index per signed offset, -1 if none
    int nwork, nkx, nky, hx;  // hx = HX (runtime); HY is the template parameter
    int bx, by, ns;           // patch, threads per patch column
};

constexpr int kHaloMax = 8;                         // positions of a patch along x and y
template <typename R> __host__ __device__ constexpr int halo_zc() { return 128 / (2 * (int)sizeof(R)); }

// Outputs a thread takes along y when ns threads share a column of a patch of `by`.
__host__ __device__ constexpr int halo_ys(int by, int ns)
{
    return (by + ns - 1) / ns < 3 ? 3 : (by + ns - 1) / ns;
}

inline size_t halo_smem(int hx, int hy, int bx, int ny, int zc, size_t elem)
{
    return ((size_t)(bx + 2 * hx) * (ny + 2 * hy) + (size_t)(2 * hx + 1) * (2 * hy + 1)) * zc * elem +
           (size_t)(bx + 2 * hx) * (ny + 2 * hy) * sizeof(int);
}

// i modulo n for i >= -n (a patch starts on the torus, and the window reaches back by
// at most n); past the second turn, which only the smallest tori have, by division.
__device__ __forceinline__ int wrap(int i, int n)
{
    i += i < 0 ? n : 0;
    i -= i >= n ? n : 0;
    return i < n ? i : i % n;
}

// MASK 1 / 2: only the source channels with a smaller / larger row index
// than the output's (V^lower / V^upper of the block Gauss-Seidel splitting,
// as k_coupling_masked); 0: the full coupling.
template <int HY, int YS, typename R, int MASK = 0>
__global__ void __launch_bounds__(4 * kHaloMax * halo_zc<R>())
k_coupling_halo(CouplingTiles ct, const int *__restrict__ gate, int n,
                const typename CT<R>::t *__restrict__ Vt, const typename CT<R>::t *__restrict__ src,
                const typename CT<R>::t *__restrict__ in0, R sgn, typename CT<R>::t *__restrict__ out)
{
    using C2 = typename CT<R>::t;
    using Mac = BoxMac<R>;
    constexpr int ZC = halo_zc<R>();
    constexpr int WY = 2 * HY + 1;
    constexpr int CW = YS + 2 * HY;              // halo values one thread keeps per column
    constexpr int E = (int)sizeof(C2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int HX = ct.hx, BX = ct.bx;
    const int HXW = BX + 2 * HX, HYW = ct.ns * YS + 2 * HY;
    const int nwin = (2 * HX + 1) * WY, npos = HXW * HYW;
    C2 *halo = reinterpret_cast<C2 *>(smem_raw);                              // [HXW][HYW][ZC]
    C2 *vw = halo + (size_t)npos * ZC;                                        // [window cell][ZC]
    int *rows = reinterpret_cast<int *>(vw + (size_t)nwin * ZC);              // [HXW][HYW]
    const int tid = threadIdx.x, nt = blockDim.x;                             // nt = BX ZC ns
    const int zl = tid % ZC, c = tid / ZC, nc = nt / ZC;
    const int z0 = blockIdx.y * ZC, z = z0 + zl;
    const int nkx = ct.nkx, nky = ct.nky;

    const int4 w = ct.work[blockIdx.x];
    const int *pr = ct.pos_row + (size_t)w.x * nkx * nky;
    if (gate && gate[w.x] == 0) return;
    // source row of every halo position (absent channels: -1)
    for (int p = tid; p < npos; p += nt) {
        const int hx = p / HYW, hy = p - hx * HYW;
        const int gx = wrap(w.y + hx - HX, nkx), gy = wrap(w.z + hy - HY, nky);
        rows[p] = pr[gx * nky + gy];
    }
    // tap values of this z range, one line per window cell (zero where no tap)
    constexpr int kU = 8;
    for (int b = c; b < nwin; b += kU * nc) {
        int t[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) t[u] = b + u * nc < nwin ? ct.tap_window[b + u * nc] : -1;
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (b + u * nc < nwin) {
                const bool ok = t[u] >= 0 && z < n;
                cp_async_zfill<E>(vw + (b + u * nc) * ZC + zl, ok ? Vt + (size_t)t[u] * n + z : Vt, ok);
            }
    }
    __syncthreads();
    if (E == 8 && (n & 1) == 0) {
        // FP32, n even: two consecutive z per 16-byte copy (z < n implies z + 1 < n)
        constexpr int ZP = ZC / 2;
        const int zp = 2 * (tid % ZP);
        const bool zok = z0 + zp < n;
#pragma unroll 4
        for (int p = tid / ZP; p < npos; p += nt / ZP) {
            const int row = rows[p];
            const bool ok = row >= 0 && zok;
            cp_async_zfill<16>(halo + p * ZC + zp, ok ? src + (size_t)row * n + z0 + zp : src, ok);
        }
    } else {
#pragma unroll 4
        for (int p = c; p < npos; p += nc) {
            const int row = rows[p];
            const bool ok = row >= 0 && z < n;
            cp_async_zfill<E>(halo + p * ZC + zl, ok ? src + (size_t)row * n + z : src, ok);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");

    const int ysub = c / BX, tx = c - ysub * BX;   // patch column, slice of its y outputs
    const int *own = rows + (tx + HX) * HYW + ysub * YS + HY;
    int rowv[YS];
    C2 base[YS];
    bool any = false;
#pragma unroll
    for (int y = 0; y < YS; ++y) {
        const int yy = ysub * YS + y;
        rowv[y] = yy < ct.by && w.z + yy < nky && w.y + tx < nkx && z < n ? own[y] : -1;
        any |= rowv[y] >= 0;
        base[y] = in0 && rowv[y] >= 0 ? in0[(size_t)rowv[y] * n + z] : mk2<R>(0, 0);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // a column of the patch without channels (the edge of a truncated set) is done
    if (!any) return;
    typename Mac::Acc acc[YS];
#pragma unroll
    for (int y = 0; y < YS; ++y) Mac::zero(acc[y]);
    for (int sdx = 0; sdx <= 2 * HX; ++sdx) {
        const int hx = tx + 2 * HX - sdx;
        const C2 *colp = halo + ((size_t)hx * HYW + ysub * YS) * ZC + zl;
        const C2 *vrow = vw + (size_t)sdx * WY * ZC + zl;
        C2 col[CW];
#pragma unroll
        for (int i = 0; i < CW; ++i) col[i] = colp[i * ZC];
        int crow[MASK ? CW : 1];
        if (MASK) {
#pragma unroll
            for (int i = 0; i < CW; ++i) crow[i] = rows[hx * HYW + ysub * YS + i];
        }
#pragma unroll
        for (int sdy = 0; sdy < WY; ++sdy) {
            const typename Mac::Tap v = Mac::tap(vrow[sdy * ZC]);
#pragma unroll
            for (int y = 0; y < YS; ++y) {
                C2 q = col[y + 2 * HY - sdy];
                if (MASK) {
                    const int sr = crow[MASK ? y + 2 * HY - sdy : 0];
                    if (!(MASK == 1 ? sr < rowv[y] : sr > rowv[y])) q = mk2<R>(0, 0);
                }
                Mac::mac(acc[y], v, Mac::val(q));
            }
        }
    }
#pragma unroll
    for (int y = 0; y < YS; ++y)
        if (rowv[y] >= 0) {
            const C2 a = Mac::get(acc[y]);
            out[(size_t)rowv[y] * n + z] = mk2<R>(base[y].x + sgn * a.x, base[y].y + sgn * a.y);
        }
}

}  // namespace msc
