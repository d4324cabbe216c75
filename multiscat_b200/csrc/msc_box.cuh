// msc_box.cuh -- channel coupling of a separable potential over whole channel boxes.
//
// Where every z's tap window factorises as V_(sdx, sdy)(z) = p_sdx(z) q_sdy(z) off
// the centre (the corrugated Morse potential of a square lattice: the FFT of
// e^{2 alpha xi} is a product of two 1-D transforms) the 2-D convolution is a
// pass along x and a pass along y:
//   t(x, y)   = sum_sdx p_sdx src(x - sdx, y)
//   out(x, y) = in0 + sgn [sum_sdy q_sdy t(x, y - sdy) - kappa src(x, y)]
// with kappa = p_0 q_0 the product's value at the centre, which is no tap.
//
// A block owns the bounding box of ONE system's channels on the torus and ZC
// consecutive z: it stages the box once in shared memory, writes t beside it, and
// runs the y pass from there, (2 H + 1) + (2 H + 2) complex MACs per box position
// with every value of src read from memory once.  (Cut into 8 x 8 patches with a halo
// on all sides, the form this replaces, a 17 x 17 box was 9 patches of 16 x 16
// positions: 8 times the loads, and the x pass ran on the y halo of every patch.)  A
// box too large for its share of shared memory is cut into strips of rows (and, past
// kBoxMaxX columns, of columns) with a halo of H.
// A thread takes SEG outputs along a line, walks the SEG + 2 H inputs once and
// keeps the 2 H + 1 taps of its z in registers: one shared-memory read per
// (2 H + 1) SEG / (SEG + 2 H) complex MACs.  Consecutive lanes are consecutive in
// z, then across the line (odd column stride: no bank conflicts).
// What bounds it: instruction issue (about half the slots go to addresses, stores and
// the gather, the rest to packed FMAs) and the latency of the gather with 24 warps
// per SM.  Measured, full batches, us, patches -> boxes: 119409 x 150 FP32 387 -> 247,
// 29856 x 150 FP64 187 -> 122, 26244 x 300 (H = 8) FP32 374 -> 203, FP64 816 -> 374
// (HBM floors 66, 33, 29 and 58); averages over a solve 194 -> 123, 118 -> 77, 247 ->
// 136 and 707 -> 330.  Tried: SEG 3 / 5 / 9 (237 / 261 / 239 against 226
// for 6 at H = 4), 128 or 448 threads (281 / 246), 16 z per block (325), bounds tests
// instead of zero margins in t (256).
#pragma once

#include <algorithm>
#include <type_traits>

#include "msc_kernels.cuh"

namespace msc {

constexpr int kBoxMaxX = 96;     // columns of a box before it is cut along x

struct BoxWork {
    int sys;
    int xh, y0;         // torus column of staged column 0 (H left of the box), first staged row
    int wx, wy;         // output columns, staged rows
    int ny;             // output rows
    int strip;          // 1: a strip of rows (wy = ny + 2 H staged, outputs start at row H); 0: wy = ny
    int wrap;           // bit 0: load the margin columns (a box around the torus, a strip of
                        // columns), else they are zero; bit 1: the box runs around the torus in y
};

struct BoxArgs {
    const BoxWork *work;
    const int *pos_row;     // [B][nkx * nky]: row of each torus position, -1 if absent
    int nkx, nky;
    int nzc;                // z chunks
    const void *p, *q;      // [2 H + 1][n] complex (R): p_sdx at sdx + H, q_sdy at sdy + H
    const void *kappa;      // [n] complex (R)
};

// Elements per z of the staged box (H margin columns on both sides, whole segments,
// odd column stride) and of t (with margin rows: H on both sides).
template <int H, int SEG>
__host__ __device__ constexpr int box_cells_s(int wx, int wy)
{
    return ((wx + SEG - 1) / SEG * SEG + 2 * H) * (wy | 1);
}
template <int H, bool TM>
__host__ __device__ constexpr int box_cells_t(int wx, int wy) { return wx * ((wy + (TM ? 2 * H : 0)) | 1); }
// Shared memory: src, t, the row of every box position, and what the last segment of
// a line may read past the end.
template <typename R, int SEG>
constexpr size_t box_smem(int cells_s, int cells_t, int zc)
{
    return (size_t)(cells_s + cells_t) * zc * 2 * sizeof(R) +
           std::max((size_t)cells_s * sizeof(int), (size_t)SEG * zc * 2 * sizeof(R));
}

// acc += tap v on complex values, kept as r += Re(tap) (vx, vy), i += Im(tap) (vx, vy)
// and combined once per output (re = r.x - i.y, im = r.y + i.x), so that a value
// needs no rotated copy.  FP32: one packed fma each (half the issue slots of the
// four scalar FMAs at the same FMA rate).
template <typename R> struct BoxMac;
template <> struct BoxMac<double> {
    struct Tap { double2 t; };
    struct Acc { double2 a; };
    using Val = double2;
    static __device__ __forceinline__ Tap tap(double2 t) { return Tap{t}; }
    static __device__ __forceinline__ Val val(double2 v) { return v; }
    static __device__ __forceinline__ void zero(Acc &c) { c.a = make_double2(0.0, 0.0); }
    static __device__ __forceinline__ void mac(Acc &c, const Tap &t, const Val &v)
    {
        c.a.x = fma(t.t.x, v.x, fma(-t.t.y, v.y, c.a.x));
        c.a.y = fma(t.t.x, v.y, fma(t.t.y, v.x, c.a.y));
    }
    static __device__ __forceinline__ double2 get(const Acc &c) { return c.a; }
};
template <> struct BoxMac<float> {
    using U = unsigned long long;
    struct Tap { U r, i; };                          // (re, re), (im, im)
    struct Acc { U r, i; };
    using Val = U;
    static __device__ __forceinline__ U pack(float x, float y)
    {
        U u;
        asm("mov.b64 %0, {%1, %2};" : "=l"(u) : "f"(x), "f"(y));
        return u;
    }
    static __device__ __forceinline__ float2 unpack(U u)
    {
        float2 f;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(u));
        return f;
    }
    static __device__ __forceinline__ Tap tap(float2 t) { return Tap{pack(t.x, t.x), pack(t.y, t.y)}; }
    static __device__ __forceinline__ Val val(float2 v) { return pack(v.x, v.y); }
    static __device__ __forceinline__ void zero(Acc &c) { c.r = c.i = 0ull; }
    static __device__ __forceinline__ void mac(Acc &c, const Tap &t, const Val &v)
    {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c.r) : "l"(t.r), "l"(v));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c.i) : "l"(t.i), "l"(v));
    }
    static __device__ __forceinline__ float2 get(const Acc &c)
    {
        const float2 r = unpack(c.r), i = unpack(c.i);
        return make_float2(r.x - i.y, r.y + i.x);
    }
};

// Asynchronous copy of BYTES (8 or 16) to shared memory; ok = false writes zeros.
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void *dst, const void *src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES),
                 "r"(ok ? BYTES : 0)
                 : "memory");
}

// Instances.  kind 0: the most z per block (whole 32- or 64-byte sectors of a row, the
// largest batches), kinds 1 and 2: half and a quarter of it (wider boxes whole or in
// fewer strips, more blocks for small batches).  MINB blocks share an SM, which sets
// the shared memory a block may take.  TM: zero or repeated margin rows in t instead
// of bounds tests (FP32, where shared memory is not what limits the blocks).
template <int H, typename R, int KIND> struct BoxShape {
    static constexpr bool wide = H > 4, f32 = sizeof(R) == 4;
    static constexpr int zc = wide ? (f32 ? (KIND == 0 ? 4 : 2) : (KIND == 0 ? 2 : 1)) : 8 >> KIND;
    static constexpr int seg = wide ? 9 : 6;
    static constexpr int nt = wide ? (f32 && KIND > 0 ? 384 : 512) : 256;
    static constexpr int minb = wide ? 1 : f32 ? 3 : 2;
    static constexpr bool tm = !wide && (f32 || KIND > 0);
    static constexpr size_t room = minb == 1 ? 227 * 1024 : (228 / minb - 2) * 1024;
    static size_t smem(int wx, int wy)           // of output columns wx and staged rows wy
    {
        return box_smem<R, seg>(box_cells_s<H, seg>(wx, wy), box_cells_t<H, tm>(wx, wy), zc);
    }
};

template <int H, int ZC, typename R, int SEG, int NT, int MINB, bool TM>
__global__ void __launch_bounds__(NT, MINB)
k_coupling_box(BoxArgs a, const int *__restrict__ gate, int n, const typename CT<R>::t *__restrict__ src,
               const typename CT<R>::t *__restrict__ in0, R sgn, typename CT<R>::t *__restrict__ out)
{
    using C2 = typename CT<R>::t;
    using M = BoxMac<R>;
    constexpr int WT = 2 * H + 1, NI = SEG + 2 * H, TH = TM ? H : 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int w = blockIdx.x / a.nzc;
    const int z0 = (blockIdx.x - w * a.nzc) * ZC;
    const BoxWork bw = a.work[w];
    if (gate && gate[bw.sys] == 0) return;
    const int wx = bw.wx, wy = bw.wy, ny = bw.ny;
    // column strides; with TM, t has H margin rows on both sides
    const int ld = (wy | 1) * ZC, tld = ((wy + 2 * TH) | 1) * ZC;
    C2 *sv = reinterpret_cast<C2 *>(smem_raw);                     // [wx + 2 H][wy | 1][ZC]
    C2 *tv = sv + box_cells_s<H, SEG>(wx, wy) * ZC;                                    // [wx][wy + 2 TH | 1][ZC]
    int *rows = reinterpret_cast<int *>(tv + box_cells_t<H, TM>(wx, wy) * ZC);        // [wx][wy]
    const int tid = threadIdx.x;
    const int zl = tid % ZC, z = z0 + zl;
    const bool zok = z < n;
    const bool margins = bw.wrap & 1;
    // ---- stage src by asynchronous copies: a group of zv lanes per position; absent
    // channels and z past n arrive as zeros.
    auto stage = [&](auto bytes) {
        constexpr int BYTES = decltype(bytes)::value;
        constexpr int EL = BYTES > (int)sizeof(C2) ? 2 : 1;  // elements per copy
        constexpr int zv = ZC / EL, step = NT / zv;
        const int zi = (tid % zv) * EL;
        const int *pr = a.pos_row + (size_t)bw.sys * a.nkx * a.nky;
        const int x_end = margins ? wx + 2 * H : wx + H;   // staged columns to copy
        const int dx = step / wy, dy = step - dx * wy;
        int x = (tid / zv) / wy, y = tid / zv - x * wy;
        x += margins ? 0 : H;
        const bool zin = z0 + zi < n;                      // EL = 2: n even, so both are
        const C2 *sp = src + z0 + zi;
        while (x < x_end) {
            int gx = bw.xh + x, gy = bw.y0 + y;
            while (gx >= a.nkx) gx -= a.nkx;
            while (gy >= a.nky) gy -= a.nky;
            const int row = __ldg(pr + gx * a.nky + gy);
            const bool ok = row >= 0 && zin;
            cp_async_zfill<BYTES>(sv + x * ld + y * ZC + zi, ok ? sp + (size_t)row * n : src, ok);
            if (zi == 0 && (unsigned)(x - H) < (unsigned)wx) rows[(x - H) * wy + y] = row;
            x += dx;
            y += dy;
            if (y >= wy) {
                y -= wy;
                ++x;
            }
        }
    };
    if constexpr (std::is_same<R, double>::value) {
        stage(std::integral_constant<int, 16>{});
    } else {
        if (n & 1) stage(std::integral_constant<int, 8>{});
        else stage(std::integral_constant<int, 16>{});
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (!margins) {
        for (int i = tid; i < H * ld; i += NT) {
            sv[i] = mk2<R>(0, 0);
            sv[(wx + H) * ld + i] = mk2<R>(0, 0);
        }
    }
    if (TM && !(bw.wrap & 2)) {
        // t margins of a box that does not run around in y
        for (int i = tid; i < wx * 2 * H * ZC; i += NT) {
            const int x = i / (2 * H * ZC), r = i - x * (2 * H * ZC);
            tv[x * tld + r + (r >= H * ZC ? wy * ZC : 0)] = mk2<R>(0, 0);
        }
    }
    // taps of this thread's z (all its items share it: the strides are multiples of ZC)
    typename M::Tap tap[WT];
    {
        const C2 *P = reinterpret_cast<const C2 *>(a.p) + (zok ? z : 0);
#pragma unroll
        for (int s = 0; s < WT; ++s) tap[s] = M::tap(__ldg(P + s * n));
    }
    // exact quotients of small numbers by wy, wx (below 2^16 here)
    const unsigned my = 0xffffffffu / (unsigned)wy + 1u, mx = 0xffffffffu / (unsigned)wx + 1u;
    auto div_y = [&](int i) { return wy == 1 ? i : (int)__umulhi((unsigned)i, my); };
    auto div_x = [&](int i) { return wx == 1 ? i : (int)__umulhi((unsigned)i, mx); };
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    const int nsy = (ny + SEG - 1) / SEG, yoff = bw.strip ? H : 0;
    // ---- x pass: items (segment, y, z)
    {
        const int nseg = (wx + SEG - 1) / SEG;
        const bool dup = bw.wrap & 2;
        for (int it = tid; it < nseg * wy * ZC; it += NT) {
            const int r = it / ZC, seg = div_y(r), y = r - seg * wy, xs = seg * SEG;
            const C2 *in = sv + xs * ld + y * ZC + zl;
            typename M::Acc acc[SEG];
#pragma unroll
            for (int o = 0; o < SEG; ++o) M::zero(acc[o]);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const typename M::Val v = M::val(*in);
                in += ld;
#pragma unroll
                for (int o = 0; o < SEG; ++o) {
                    const int s = o + 2 * H - i;           // tap index sdx + H
                    if (s >= 0 && s < WT) M::mac(acc[o], tap[s], v);
                }
            }
            C2 *to = tv + xs * tld + (y + TH) * ZC + zl;
            const int nv = min(SEG, wx - xs);
#pragma unroll
            for (int o = 0; o < SEG; ++o) {
                if (o < nv) *to = M::get(acc[o]);
                to += tld;
            }
            if (TM && dup && (y < H || y >= wy - H)) {
                // rows that a box running around in y repeats on its other side
                to -= SEG * tld;
                for (int o = 0; o < nv; ++o, to += tld) {
                    const C2 v = *to;
                    if (y >= wy - H) to[-wy * ZC] = v;
                    if (y < H) to[wy * ZC] = v;
                }
            }
        }
    }
    typename M::Tap ktap;
    {
        const C2 *Q = reinterpret_cast<const C2 *>(a.q) + (zok ? z : 0);
#pragma unroll
        for (int s = 0; s < WT; ++s) tap[s] = M::tap(__ldg(Q + s * n));
        const C2 k = __ldg(reinterpret_cast<const C2 *>(a.kappa) + (zok ? z : 0));
        ktap = M::tap(mk2<R>(-k.x, -k.y));
    }
    __syncthreads();

    // ---- y pass: items (segment, x, z); segments without a channel are skipped
    const bool wrapy = bw.wrap & 2;
    for (int it = tid; it < nsy * wx * ZC; it += NT) {
        const int r = it / ZC, seg = div_x(r), x = r - seg * wx, ys = seg * SEG, y0 = yoff + ys;
        const int *rp = rows + x * wy + y0;
        int rowv[SEG];
        bool any = false;
#pragma unroll
        for (int o = 0; o < SEG; ++o) {
            rowv[o] = ys + o < ny ? rp[o] : -1;
            any |= rowv[o] >= 0;
        }
        if (!any || !zok) continue;
        C2 base[SEG];
#pragma unroll
        for (int o = 0; o < SEG; ++o)
            base[o] = (in0 && rowv[o] >= 0) ? in0[(size_t)rowv[o] * n + z] : mk2<R>(0, 0);
        const C2 *own = sv + (x + H) * ld + y0 * ZC + zl;
        const C2 *in = tv + x * tld + zl + (TM ? y0 * ZC : 0);
        typename M::Acc acc[SEG];
#pragma unroll
        for (int o = 0; o < SEG; ++o) {
            M::zero(acc[o]);
            M::mac(acc[o], ktap, M::val(own[o * ZC]));
        }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            typename M::Val v;
            if constexpr (TM) {
                v = M::val(in[i * ZC]);
            } else {
                int y = y0 + i - H;
                if (wrapy) y += y < 0 ? wy : y >= wy ? -wy : 0;
                v = M::val((unsigned)y < (unsigned)wy ? in[y * ZC] : mk2<R>(0, 0));
            }
#pragma unroll
            for (int o = 0; o < SEG; ++o) {
                const int s = o + 2 * H - i;
                if (s >= 0 && s < WT) M::mac(acc[o], tap[s], v);
            }
        }
#pragma unroll
        for (int o = 0; o < SEG; ++o)
            if (rowv[o] >= 0) {
                const C2 v = M::get(acc[o]);
                out[(size_t)rowv[o] * n + z] = mk2<R>(base[o].x + sgn * v.x, base[o].y + sgn * v.y);
            }
    }
}

}  // namespace msc
