// msc_eigh_gpu.cuh -- FP64 symmetric eigen-decomposition of H0 on the GPU.
//
// The preconditioner needs H0 = T + diag Re V_00 = E diag(lam) E^T once per
// potential (the reference: build_preconditioner, multiscat_gmres.f90:226-273,
// with EISPACK rs = tred2 + tql2, diagsub.f90:5-262).  Here the O(n^3) parts
// run on the device and the host does O(n^2) scalar work only:
//
//   1. k_tridiagonalize (one CTA) or k_tridiagonalize_cluster (8 or 16 CTAs, the
//      rows dealt out over their shared memories): Householder reduction
//      A = Q_H T Q_H^T, Q_H = H_0 H_1 ... H_{n-3}, H_k = I - 2 v_k v_k^T (unit v_k
//      supported on k+1 .. n-1).
//   2. host: implicit symmetric QR with Wilkinson shifts on the tridiagonal
//      (d, e), recording every Givens rotation (k, c, s) it applies
//      (tridiagonal_qr_rotations in msc_eigh.hpp).  O(n) per sweep.
//   3. k_apply_rotations: Z = G_1 G_2 ... from the identity, one thread per
//      row of Z; a rotation acts on columns k, k+1 of every row, so rows are
//      independent and each CTA keeps its rows in shared memory.
//   4. k_back_transform: E = Q_H Z, the reflectors applied from the left in
//      reverse order; a reflector acts on rows, so columns are independent
//      and each warp keeps its columns in registers.  Columns are written
//      in ascending eigenvalue order.
//
// All three are chains of n (or 0.9 n^2 rotations) dependent steps, so latency per
// step is what bounds them.  Measured, ms, n = 100 / 550 (before -> now): reduction
// 0.45 / 36 -> 0.2 / 3.6, rotations 0.68 / 19 -> 0.1 / 3.3, back-transformation 0.19 /
// 2.1 -> 0.03 / 0.29; whole decomposition with the host's iteration and the copies, n =
// 100 / 200 / 300 / 550: 1.7 / 6.2 / 15.3 / 65 -> 0.9 / 2.4 / 4.9 / 14.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "msc_common.cuh"

namespace msc {
namespace eig {

constexpr int kTriThreads = 1024;
constexpr int kTriSmemMaxN = 160;          // n^2 doubles in one CTA's shared memory up to here

// One step's scalars from x (the column below the diagonal, m entries), y = S x and
// s0 = row 0 of S, found by every warp for itself (same order, same result):
//   alpha = -sign(x_0) |x|,  v = (x - alpha e_0) inv,  S v = (y - alpha s0) inv,
//   v^T S v = inv^2 (x^T y - 2 alpha y_0 + alpha^2 S_00)
// so that the product with S needs x only and runs before the norm is known.  alpha
// has the sign opposite to x_0: nothing cancels in x_0 - alpha or y - alpha s0.
// (x^T y and the terms beside it are of third order in the matrix: the caller keeps its
// largest entry between 2^-200 and 2^200 by a power of two.)
struct TriStep {
    double alpha, inv, vp;
    bool applied;
};

__device__ __forceinline__ TriStep tri_step(int m, const double *x, const double *y, const double *s0, int lane)
{
    double n2 = 0.0, xy = 0.0;
    for (int i = lane; i < m; i += 32) {
        n2 = fma(x[i], x[i], n2);
        xy = fma(x[i], y[i], xy);
    }
    n2 = warp_sum(n2);
    xy = warp_sum(xy);
    TriStep t{};
    t.applied = n2 != 0.0;
    if (t.applied) {
        const double x0 = x[0];
        t.alpha = (x0 >= 0.0) ? -sqrt(n2) : sqrt(n2);
        t.inv = 1.0 / sqrt(n2 - x0 * x0 + (x0 - t.alpha) * (x0 - t.alpha));
        t.vp = t.inv * (t.inv * (xy - 2.0 * t.alpha * y[0] + t.alpha * t.alpha * s0[0]));
    }
    return t;
}

// A: n x n symmetric, row-major, full storage (destroyed).  R: row k holds
// v_k at columns k+1 .. n-1 (unit vector); applied[k] = 0 when column k
// needed no reflection.  d[n], e[n-1].  Dynamic shared memory: five vectors, after
// the matrix itself when n <= kTriSmemMaxN.
__host__ __device__ constexpr size_t tri_smem(int n)
{
    return ((n <= kTriSmemMaxN ? (size_t)n * n : 0) + (size_t)5 * n) * sizeof(double);
}
// Three block barriers a step (product, vectors, rank-2 update); nine before.
__global__ void __launch_bounds__(kTriThreads)
k_tridiagonalize(int n, double *__restrict__ A, double *__restrict__ R, double *__restrict__ d,
                 double *__restrict__ e, int *__restrict__ applied)
{
    extern __shared__ double sm_a[];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    const bool in_smem = n <= kTriSmemMaxN;
    double *v = sm_a + (in_smem ? n * n : 0), *p = v + n, *xs = p + n, *ys = xs + n, *s0 = ys + n;
    double *M = A;
    if (in_smem) {
        for (int i = tid; i < n * n; i += nt) sm_a[i] = A[i];
        M = sm_a;
        __syncthreads();
    }
    for (int k = 0; k + 2 < n; ++k) {
        const int m = n - k - 1;
        const double *x = M + (size_t)k * n + (k + 1);       // = column k below the diagonal
        const double *S = M + (size_t)(k + 1) * n + (k + 1);
        for (int i = warp; i < m; i += nw) {
            const double *row = S + (size_t)i * n;
            double s = 0.0;
            for (int j = lane; j < m; j += 32) s = fma(row[j], x[j], s);
            s = warp_sum(s);
            if (lane == 0) ys[i] = s;
        }
        for (int i = tid; i < m; i += nt) {
            xs[i] = x[i];
            s0[i] = S[i];
        }
        __syncthreads();
        const TriStep t = tri_step(m, xs, ys, s0, lane);
        if (t.applied) {
            for (int i = tid; i < m; i += nt) {
                const double vi = (i == 0 ? xs[0] - t.alpha : xs[i]) * t.inv;
                v[i] = vi;
                p[i] = (ys[i] - t.alpha * s0[i]) * t.inv - t.vp * vi;
                R[(size_t)k * n + (k + 1) + i] = vi;
            }
        }
        if (tid == 0) {
            d[k] = M[(size_t)k * n + k];
            e[k] = t.alpha;
            applied[k] = t.applied;
        }
        __syncthreads();
        if (!t.applied) continue;
        // S <- (I - 2 v v^T) S (I - 2 v v^T) = S - 2 v p^T - 2 p v^T
        for (int i = warp; i < m; i += nw) {
            double *row = M + (size_t)(k + 1 + i) * n + (k + 1);
            const double vi2 = 2.0 * v[i], pi2 = 2.0 * p[i];
            for (int j = lane; j < m; j += 32) row[j] -= vi2 * p[j] + pi2 * v[j];
        }
        __syncthreads();
    }
    if (tid == 0) {
        if (n >= 2) {
            d[n - 2] = M[(size_t)(n - 2) * n + (n - 2)];
            e[n - 2] = M[(size_t)(n - 1) * n + (n - 2)];
            applied[n - 2] = 0;
        }
        d[n - 1] = M[(size_t)(n - 1) * n + (n - 1)];
        applied[n - 1] = 0;
    }
}

// The same reduction with row i in the shared memory of CTA i mod CL of one cluster
// (n > 160: one SM reading the matrix three times a step from L2 was 65 us a step at
// n = 550).  Per step every CTA forms its rows of y = S x and sends them to all; all
// form v and p; each updates its rows, and the owners of the next two rows (the next
// x and s0) send those.  Two cluster barriers a step.  Grid: one cluster of CL CTAs.
__host__ __device__ constexpr size_t tri_cluster_smem(int n, int cl)
{
    // rows, then y, v, p, and x and s0 twice (read and written in the same phase)
    return ((size_t)((n + cl - 1) / cl) * n + (size_t)7 * n) * sizeof(double);
}

__global__ void __launch_bounds__(kTriThreads)
k_tridiagonalize_cluster(int n, const double *__restrict__ A, double *__restrict__ R, double *__restrict__ d,
                         double *__restrict__ e, int *__restrict__ applied)
{
    namespace cg = cooperative_groups;
    extern __shared__ double sm_a[];
    const cg::cluster_group cluster = cg::this_cluster();
    const int cl = (int)cluster.num_blocks(), c = (int)cluster.block_rank();
    const int nloc = (n + cl - 1) / cl;
    double *M = sm_a;                                   // [nloc][n]: rows c, c + cl, ...
    double *ys = M + (size_t)nloc * n, *v = ys + n, *p = v + n;
    double *xb = p + n, *sb = xb + 2 * n;               // [2][n] each: x and s0 of even / odd steps
    const int tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    for (int i = tid; i < nloc * n; i += nt) {
        const int r = i / n, row = c + r * cl;
        M[i] = row < n ? A[(size_t)row * n + (i - r * n)] : 0.0;
    }
    for (int i = tid; i < n; i += nt) {                 // rows 0 and 1, whole (indexed by column)
        xb[i] = A[i];
        sb[i] = A[n + i];
    }
    cluster.sync();
    for (int k = 0; k + 2 < n; ++k) {
        const int m = n - k - 1, par = k & 1;
        const double *x = xb + (size_t)par * n + (k + 1), *s0 = sb + (size_t)par * n + (k + 1);
        // first local row with index > k
        const int r0 = k + 1 <= c ? 0 : (k + 1 - c + cl - 1) / cl;
        for (int r = r0 + warp; r < nloc; r += nw) {
            const int row = c + r * cl;
            if (row >= n) break;
            const double *mr = M + (size_t)r * n + (k + 1);
            double s = 0.0;
            for (int j = lane; j < m; j += 32) s = fma(mr[j], x[j], s);
            s = warp_sum(s);
            if (lane < cl) cluster.map_shared_rank(ys, lane)[row - (k + 1)] = s;
        }
        cluster.sync();
        const TriStep t = tri_step(m, x, ys, s0, lane);
        for (int i = tid; i < m; i += nt) {
            const double vi = t.applied ? (i == 0 ? x[0] - t.alpha : x[i]) * t.inv : 0.0;
            v[i] = vi;
            p[i] = t.applied ? (ys[i] - t.alpha * s0[i]) * t.inv - t.vp * vi : 0.0;
            if (c == 0 && t.applied) R[(size_t)k * n + (k + 1) + i] = vi;
        }
        if (c == 0 && tid == 0) {
            d[k] = xb[(size_t)par * n + k];
            e[k] = t.alpha;
            applied[k] = t.applied;
        }
        __syncthreads();
        double *xn = xb + (size_t)(par ^ 1) * n, *sn = sb + (size_t)(par ^ 1) * n;
        for (int r = r0 + warp; r < nloc; r += nw) {
            const int row = c + r * cl;
            if (row >= n) break;
            double *mr = M + (size_t)r * n + (k + 1);
            const double vi2 = 2.0 * v[row - (k + 1)], pi2 = 2.0 * p[row - (k + 1)];
            double *send = row == k + 1 ? xn : row == k + 2 ? sn : nullptr;   // the next x, s0
            for (int j = lane; j < m; j += 32) {
                const double u = mr[j] - (vi2 * p[j] + pi2 * v[j]);
                mr[j] = u;
                if (send)
                    for (int q = 0; q < cl; ++q) cluster.map_shared_rank(send, q)[k + 1 + j] = u;
            }
        }
        cluster.sync();     // rows in place everywhere; y, v and p may be rewritten
    }
    // the last 2 x 2 block: rows n - 2 and n - 1 are the current x and s0 buffers
    if (c == 0 && tid == 0) {
        const int par = (n - 2) & 1;
        const double *x = xb + (size_t)par * n, *s0 = sb + (size_t)par * n;
        d[n - 2] = x[n - 2];
        e[n - 2] = s0[n - 2];
        d[n - 1] = s0[n - 1];
        applied[n - 2] = applied[n - 1] = 0;
    }
}

// Z = G_1 G_2 ... G_r (from the identity): rotation (k, c, s) acts on columns
// k, k + 1 of every row: (z_k, z_{k+1}) <- (c z_k + s z_{k+1}, c z_{k+1} - s z_k).
// One thread per row, RB rows per CTA kept in shared memory as zs[col][row].
// The rotations come in sweeps of rising k; four sweeps run through a row together,
// each two columns behind the one before it: sweep j takes column k + 1 from sweep
// j - 1's output of the step before, so a step is four independent rotations (one
// chain of one fma each) and the row passes through shared memory once per four
// sweeps.  tab[step][4] holds the coefficients (c, s) of a step, already skewed,
// groups (lo, hi, first step) the column ranges; sweeps are padded to their group's
// range with identity rotations.  (One rotation at a time with its operands from L2:
// 150 cycles each; n = 100: 680 us.)  Output Zt[col][row] (column-major Z).
// The table is one stream (the groups' steps follow one another): it arrives by
// asynchronous copies, kRotChunk steps ahead of their use.
constexpr int kRotChunk = 64;
template <int RB>
__host__ __device__ constexpr size_t rotations_smem(int n)
{
    return (size_t)n * RB * sizeof(double) + (size_t)3 * kRotChunk * 4 * sizeof(double2);
}

template <int RB>
__global__ void __launch_bounds__(32)
k_apply_rotations(int n, int ngroups, int nsteps, const int4 *__restrict__ groups,
                  const double2 *__restrict__ tab, double *__restrict__ Zt)
{
    extern __shared__ __align__(16) double zs_all[];
    double2 *ring = reinterpret_cast<double2 *>(zs_all);      // [3][kRotChunk][4]
    double *zs = zs_all + (size_t)3 * kRotChunk * 8;          // [n][RB]
    const int t = threadIdx.x % RB;                           // (RB = 16: lanes 16.. read as 0..15, write nothing)
    const int row = blockIdx.x * RB + t;
    const bool own = threadIdx.x < RB;                        // one lane writes a cell
    if (own)
        for (int c = 0; c < n; ++c) zs[c * RB + t] = (c == row) ? 1.0 : 0.0;
    __syncwarp();
    // chunk q of the table into ring slot q % 3; past the end nothing is copied
    auto fetch = [&](int q) {
        const int lo = q * kRotChunk * 4, hi = min(nsteps, (q + 1) * kRotChunk) * 4;
        double2 *dst = ring + (size_t)(q % 3) * kRotChunk * 4;
        for (int i = lo + (int)threadIdx.x; i < hi; i += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + (i - lo))), "l"(tab + i)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    fetch(1);
    int pos = 0;                                              // step of the whole table
    int4 gr = ngroups > 0 ? __ldg(groups) : make_int4(0, 0, 0, 0);
    for (int g = 0; g < ngroups; ++g) {
        const int4 gnext = __ldg(groups + min(g + 1, ngroups - 1));
        const int lo = gr.x, L = gr.y - gr.x;
        double carry[4], o1[4], o2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) carry[j] = o1[j] = o2[j] = 0.0;
        double znext = zs[(lo + 1) * RB + t];
        carry[0] = zs[lo * RB + t];
        // one step; EDGE: some sweep is outside its range (the first 7 steps and the last 6)
        auto step = [&](int st, const double2 *cs, auto edge) {
            constexpr bool EDGE = decltype(edge)::value;
            const double zin = znext;
            if (!EDGE || st + 1 < L) znext = zs[min(lo + st + 2, n - 1) * RB + t];
            double on[4];
#pragma unroll
            for (int j = 3; j >= 0; --j) {         // from the last: sweep j reads j - 1's old state
                const int i = st - 2 * j;
                on[j] = 0.0;
                if (EDGE && (i < 0 || i >= L)) continue;
                const double2 r = cs[j];
                if (EDGE && j > 0 && i == 0) carry[j] = o2[j - 1];
                const double qb = j == 0 ? zin : !EDGE || i + 1 < L ? o1[j - 1] : carry[j - 1];
                on[j] = fma(r.x, carry[j], r.y * qb);
                carry[j] = fma(-r.y, carry[j], r.x * qb);
            }
            if (own && (!EDGE || st >= 6)) zs[(lo + st - 6) * RB + t] = on[3];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (EDGE) o2[j] = o1[j];
                o1[j] = on[j];
            }
        };
        for (int st = 0; st < L + 6;) {
            if (pos % kRotChunk == 0) {
                // the next chunk but one is requested while this one is used, into the slot
                // of the chunk before it, which every lane has to be done with
                __syncwarp();
                fetch(pos / kRotChunk + 2);
                asm volatile("cp.async.wait_group 2;" ::: "memory");
                __syncwarp();
            }
            const int run = min(L + 6 - st, kRotChunk - pos % kRotChunk);
            const double2 *cs = ring + (size_t)(pos / kRotChunk % 3) * kRotChunk * 4 + (pos % kRotChunk) * 4;
            const int end = st + run;
            for (; st < min(end, 7); ++st, cs += 4) step(st, cs, std::true_type{});
#pragma unroll 2
            for (; st < min(end, L - 1); ++st, cs += 4) step(st, cs, std::false_type{});
            for (; st < end; ++st, cs += 4) step(st, cs, std::true_type{});
            pos += run;
        }
        if (own) zs[(lo + L) * RB + t] = carry[3];
        gr = gnext;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (row < n && own)
        for (int c = 0; c < n; ++c) Zt[(size_t)c * n + row] = zs[c * RB + t];
}

// E = Q_H Z: reflectors H_{n-3} .. H_0 applied in turn (z <- z - 2 v (v^T z) on rows
// k+1 .. n-1) to CB columns of Z per warp, held in registers (NE entries a lane: rows
// lane, lane + 32, ...), the next reflector on its way while one is applied; no
// barriers (a block used to share each v through shared memory: 2 us a reflector).
// R is zero at columns <= k, so a reflector's untouched rows need no test.  Column j
// of the result is written to column dest[j] of the row-major output E[row * n + col]
// (ascending eigenvalue order).
template <int NE, int CB>
__global__ void __launch_bounds__(128)
k_back_transform(int n, const double *__restrict__ R, const int *__restrict__ applied,
                 const double *__restrict__ Zt, const int *__restrict__ dest, double *__restrict__ E)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = (blockIdx.x * 4 + warp) * CB;
    if (c0 >= n) return;
    double z[CB][NE], v[NE], vn[NE];
#pragma unroll
    for (int b = 0; b < CB; ++b)
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int r = lane + 32 * i;
            z[b][i] = c0 + b < n && r < n ? Zt[(size_t)(c0 + b) * n + r] : 0.0;
        }
    auto load = [&](int k, double (&u)[NE]) {
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int r = lane + 32 * i;
            u[i] = k >= 0 && r < n ? __ldg(R + (size_t)k * n + r) : 0.0;
        }
    };
    load(n - 3, v);
    for (int k = n - 3; k >= 0; --k) {
        load(k - 1, vn);
        if (__ldg(applied + k)) {
#pragma unroll
            for (int b = 0; b < CB; ++b) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < NE; ++i) s = fma(v[i], z[b][i], s);
                s = 2.0 * warp_sum(s);
#pragma unroll
                for (int i = 0; i < NE; ++i) z[b][i] = fma(-s, v[i], z[b][i]);
            }
        }
#pragma unroll
        for (int i = 0; i < NE; ++i) v[i] = vn[i];
    }
#pragma unroll
    for (int b = 0; b < CB; ++b)
        if (c0 + b < n) {
            const int col = dest[c0 + b];
#pragma unroll
            for (int i = 0; i < NE; ++i) {
                const int r = lane + 32 * i;
                if (r < n) E[(size_t)r * n + col] = z[b][i];
            }
        }
}

}  // namespace eig
}  // namespace msc
