// cf_box.cuh -- K3+K4, plain form: the collaborative filter of B = 8 groups with the image region of
// a tile of groups held in shared memory.
//
// A CTA takes one plane of a tile of neighbouring reference blocks.  Every block their lists
// can name lies in one box of the image, the union of their search windows, or is the block at (0, 0)
// (the reference's trailing candidate), which gets a slot of its own beside the box.  The box is
// copied to shared memory once, the groups' blocks are read from there, and their estimates are added
// into a second box in fixed point, which goes to the numerator plane once, with vector atomics.
// Shared-memory atomics are native for 32-bit integers only (float and 64-bit ones are compare-and-swap
// loops, 437 clocks a block and warp against 100), so a cell is two words of its own: a term is split
// into a multiple of 2^-13 and the rest, rounded to a multiple of 2^-32 (terms from 2^-9 on lose nothing).
//
// Final (cf_box_kernel): a pair of warps per slot of 32 blocks (32 / G groups), both filtering the
// reference and the source blocks at once as the halves of packed fp32 pairs (one instruction for
// both, each half rounded as the scalar instruction would).  2-D transforms: two lanes per block, four
// rows each, exchanged by shuffles for the columns; z stage: lane = coefficient column of the transpose
// buffer; the estimates are inverted and scattered by the warp that holds their blocks.
// The arithmetic is that of common.cuh's transforms, operation for operation, as in cf_fast_kernel.
// Bound: the FP32 pipe (9.9 k clocks of a step's 19 k; the transforms are separable butterflies, and a
// packed instruction takes the pipe twice) and, in the phases that do not use it, the latency of 16
// warps per SM, which the transpose buffers and 128 registers a thread allow.  1920x1080 RGB x 8,
// G = 32: 120.3 ms with one warp per group, gathers from global memory and a 64-bit box, 44.1 ms now.
#pragma once

#include "cf.cuh"
#include "tc.cuh"

namespace bm3d {

// Fixed point: units of the high and the low word.  A pixel takes at most 128 groups x 32 blocks = 2^12
// terms per tile; terms below 2^6 keep the high word below 2^31 and the low one below 2^30, larger ones
// go to the plane directly.
constexpr float kBoxMax = 64.0f;
constexpr float kBoxHi = 8192.0f, kBoxHiUnit = 1.220703125e-4f;               // 2^13, 2^-13
constexpr float kBoxLo = 4294967296.0f, kBoxLoUnit = 2.3283064365386963e-10f;  // 2^32, 2^-32
constexpr float kBoxRound = 12582912.0f;                                       // 1.5 x 2^23: rounds to an integer
constexpr int kBoxRoundBits = 0x4b400000;

// sum of a cell's words as a float
__device__ __forceinline__ float box_value(int hi, int lo)
{
    // carry into the high word: the low one is then exact in fp32, the high one below 2^24 units, a sum of 2^11
    // (a larger one is rounded twice)
    return __fmaf_rn(__int2float_rn(lo & 0x7ffff), kBoxLoUnit, __int2float_rn(hi + (lo >> 19)) * kBoxHiUnit);
}

__device__ __forceinline__ void pair_barrier(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

using tc::f2;
using tc::pk;
using tc::upk;
using tc::fma2;

__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Product of both halves by scalar multiplications, for a product that a packed sum follows: a packed
// one would be contracted with the sum into one rounding
__device__ __forceinline__ f2 mul2s(f2 v, float c)
{
    float a, b;
    upk(v, a, b);
    return pk(__fmul_rn(a, c), __fmul_rn(b, c));
}

// Outputs formed together: their chains of dependent multiply-adds run side by side
constexpr int kChains = 4;

// fdct_reg on packed pairs; outputs are handed to f(k, step, X) in sets as they are produced (X[i] is
// output k + i * step), the odd ones of the longest level first, so that a column's inputs are dead
// before its spectrum is complete
template <int N, int S = 1, class F>
__device__ __forceinline__ void fdct2(const f2 (&x)[N], F &&f)
{
    if constexpr (N == 2) {
        const f2 X[2] = {tc::mul2(add2(x[0], x[1]), pk(2.0f, 2.0f)), mul2s(sub2(x[0], x[1]), odd_coef(2, 0, 0))};
        f(0, S, X);
    } else if constexpr (N == 1) {
        const f2 X[1] = {tc::mul2(x[0], pk(2.0f, 2.0f))};
        f(0, S, X);
    } else {
        constexpr int h = N / 2, C = h < kChains ? h : kChains;
        f2 e[h], o[h];
#pragma unroll
        for (int j = 0; j < h; ++j) {
            e[j] = add2(x[j], x[N - 1 - j]);
            o[j] = sub2(x[j], x[N - 1 - j]);
        }
#pragma unroll
        for (int m = 0; m < h; m += C) {
            f2 X[C];
#pragma unroll
            for (int i = 0; i < C; ++i) X[i] = tc::mul2(o[0], pk(odd_coef(N, m + i, 0), odd_coef(N, m + i, 0)));
#pragma unroll
            for (int j = 1; j < h; ++j)
#pragma unroll
                for (int i = 0; i < C; ++i) X[i] = fma2(o[j], pk(odd_coef(N, m + i, j), odd_coef(N, m + i, j)), X[i]);
            f((2 * m + 1) * S, 2 * S, X);
        }
        fdct2<h, 2 * S>(e, f);
    }
}

// idct_reg on packed pairs
template <int N>
__device__ __forceinline__ void idct2(const f2 (&X)[N], f2 (&y)[N])
{
    if constexpr (N == 2) {
        const f2 o = mul2s(X[1], odd_coef(2, 0, 0));
        y[0] = add2(X[0], o);
        y[1] = sub2(X[0], o);
    } else {
        constexpr int h = N / 2;
        f2 ev[h], E[h], o[h];
#pragma unroll
        for (int m = 0; m < h; ++m) ev[m] = X[2 * m];
        idct2<h>(ev, E);
#pragma unroll
        for (int k = 0; k < h; ++k) o[k] = tc::mul2(X[1], pk(odd_coef(N, k, 0), odd_coef(N, k, 0)));
#pragma unroll
        for (int m = 1; m < h; ++m)
#pragma unroll
            for (int k = 0; k < h; ++k) o[k] = fma2(X[2 * m + 1], pk(odd_coef(N, k, m), odd_coef(N, k, m)), o[k]);
#pragma unroll
        for (int k = 0; k < h; ++k) {
            y[k] = add2(E[k], o[k]);
            y[N - 1 - k] = sub2(E[k], o[k]);
        }
    }
}

// idct_reg with kChains outputs side by side, handed to f(k, y_k)
template <int N, class F>
__device__ __forceinline__ void idct_sets(const float (&X)[N], F &&f)
{
    if constexpr (N == 1) {
        f(0, X[0]);
    } else {
        constexpr int h = N / 2, C = h < kChains ? h : kChains;
        float ev[h], E[h];
#pragma unroll
        for (int m = 0; m < h; ++m) ev[m] = X[2 * m];
        idct_sets<h>(ev, [&](int k, float v) { E[k] = v; });
#pragma unroll
        for (int k = 0; k < h; k += C) {
            float o[C];
#pragma unroll
            for (int i = 0; i < C; ++i) o[i] = __fmul_rn(X[1], odd_coef(N, k + i, 0));
#pragma unroll
            for (int m = 1; m < h; ++m)
#pragma unroll
                for (int i = 0; i < C; ++i) o[i] = __fmaf_rn(X[2 * m + 1], odd_coef(N, k + i, m), o[i]);
#pragma unroll
            for (int i = 0; i < C; ++i) {
                f(k + i, __fadd_rn(E[k + i], o[i]));
                f(N - 1 - k - i, __fsub_rn(E[k + i], o[i]));
            }
        }
    }
}

// Wiener weights w[i] = r2[i] / (r2[i] + sg): reciprocal estimate, quotient, and one correction by the
// remainder (Markstein, IBM J. Res. Dev. 34, 1990), which rounds as the division does but for quotients
// within 2^-45 of a tie (of 4 M random pairs, none to a few, by one unit), as long as the remainder is exact: for
// r2 from 2^-102 on.  Below, the quotient stays within three units.
// EXACT: the division itself, a dozen instructions and a branch each.  A column takes it
// - where a divisor reaches 2^126 and its estimate underflows: `top` collects the largest, and the column is redone;
// - where sg is below kWienerLow, so that an r2 below 2^-102 may have a weight that counts (else it is below 2^-42):
//   `top` starts at wiener_top(sg), the limit.
constexpr float kWienerTop = 4.2535296e37f;       // 2^125
constexpr float kWienerLow = 8.6736174e-19f;      // 2^-60
__device__ __forceinline__ float wiener_top(float sg) { return sg < kWienerLow ? kWienerTop : 0.0f; }

template <bool EXACT, int C>
__device__ __forceinline__ void wiener_weights(const float (&r2)[C], float sg, float (&w)[C], float &top)
{
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const float d = __fadd_rn(r2[i], sg);
        if constexpr (EXACT) {
            w[i] = __fdiv_rn(r2[i], d);
        } else {
            top = fmaxf(top, d);
            float y;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
            const float q = __fmul_rn(r2[i], y);
            w[i] = __fmaf_rn(__fmaf_rn(-d, q, r2[i]), y, q);
        }
    }
}

// A column of N (reference, source) cells filtered by its Wiener weights: its spectrum in Y; returns the sum of
// the squared weights
template <int N, bool EXACT>
__device__ __forceinline__ float wiener_spectrum(const f2 (&x)[N], float sg, float (&Y)[N], float &top)
{
    float l2 = 0.0f;
    fdct2<N>(x, [&](int k, int st, const auto &v) {
        constexpr int C = (int)(sizeof(v) / sizeof(v[0]));
        float r2[C], sv[C], w[C];
#pragma unroll
        for (int i = 0; i < C; ++i) {
            float r;
            upk(v[i], r, sv[i]);
            r2[i] = __fmul_rn(r, r);
        }
        wiener_weights<EXACT, C>(r2, sg, w, top);
#pragma unroll
        for (int i = 0; i < C; ++i) {
            Y[k + i * st] = __fmul_rn(sv[i], w[i]);
            l2 = __fmaf_rn(w[i], w[i], l2);
        }
    });
    return l2;
}

// Z stage of a column of N cells (stride in cells), the filtered source into the cells' low words
template <int N, bool EXACT>
__device__ __forceinline__ float wiener_column(f2 *t, int stride, float sg, float &top)
{
    f2 x[N];
    float Y[N];
#pragma unroll
    for (int z = 0; z < N; ++z) x[z] = t[z * stride];
    const float l2 = wiener_spectrum<N, EXACT>(x, sg, Y, top);
    if (EXACT || top < kWienerTop) idct_sets<N>(Y, [&](int z, float v) { *reinterpret_cast<float *>(t + z * stride) = v; });
    return l2;
}

// out of line: huge values only
template <int N>
__device__ __noinline__ float wiener_column_exact(f2 *t, int stride, float sg)
{
    float top = 0.0f;
    return wiener_column<N, true>(t, stride, sg, top);
}

constexpr int kBT = 66;                  // cells between the blocks of the transpose buffer: 2 mod 16, so that
                                         // eight blocks x two columns, or 16 columns, fall in distinct banks

__device__ __forceinline__ f2 shfl_pair(f2 v)
{
    float a, b;
    upk(v, a, b);
    return pk(__shfl_xor_sync(0xffffffffu, a, 1), __shfl_xor_sync(0xffffffffu, b, 1));
}

// A block's pixels, load(y, x) -> its 2-D coefficients at `t`.  Lane half h (lane & 1) transforms rows 0 .. 3
// (h = 0) or 7 .. 4 (h = 1), then the columns 2k + h; load(i, x) gives pixel x of the lane's i-th row.
template <class Load>
__device__ __forceinline__ void box_forward(Load &&load, f2 *t, int h)
{
    f2 keep[4][4], give[4][4];            // [row][column pair]: columns 2k + h, columns 2k + 1 - h
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f2 x[8], X[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = load(i, k);
        fdct2<8>(x, [&](int k, int st, const auto &v) {
#pragma unroll
            for (int c = 0; c < (int)(sizeof(v) / sizeof(v[0])); ++c) X[k + c * st] = v[c];
        });
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            keep[i][k] = h ? X[2 * k + 1] : X[2 * k];
            give[i][k] = h ? X[2 * k] : X[2 * k + 1];
        }
    }
    const f2 sg = h ? pk(-1.0f, -1.0f) : pk(1.0f, 1.0f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        // first level of the column transform across the two lanes: lane 1's differences, and so its
        // odd outputs, have the other sign
        f2 e[4], o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f2 v = shfl_pair(give[i][k]);
            e[i] = add2(keep[i][k], v);
            o[i] = sub2(keep[i][k], v);
        }
        f2 *c = t + 2 * k + h;
        f2 X[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) X[m] = tc::mul2(o[0], pk(odd_coef(8, m, 0), odd_coef(8, m, 0)));
#pragma unroll
        for (int j = 1; j < 4; ++j)
#pragma unroll
            for (int m = 0; m < 4; ++m) X[m] = fma2(o[j], pk(odd_coef(8, m, j), odd_coef(8, m, j)), X[m]);
#pragma unroll
        for (int m = 0; m < 4; ++m) c[(2 * m + 1) * 8] = tc::mul2(X[m], sg);
        fdct2<4, 2>(e, [&](int y, int st, const auto &v) {
#pragma unroll
            for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) c[(y + i * st) * 8] = v[i];
        });
    }
}

// Inverse 2-D transform, scaled, of the filtered coefficients (the low words of the cells) of the block
// at `t`; the estimates (zeros for a place past the group's end) go to the block's first 64 words, column by column.  Lane half h inverts the
// columns 2k + h, then the rows 4h .. 4h + 3.
__device__ __forceinline__ void box_inverse(float *t, float scale, bool active, int h)
{
    float keep[4][4], give[4][4];         // [row][column k]
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        f2 X[8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) X[i] = pk(t[2 * (i * 8 + 4 * q + h)], t[2 * (i * 8 + 4 * q + 2 + h)]);
        idct2<8>(X, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a0, a1, b0, b1;
            upk(y[i], a0, a1);
            upk(y[i + 4], b0, b1);
            keep[i][2 * q] = h ? b0 : a0;
            keep[i][2 * q + 1] = h ? b1 : a1;
            give[i][2 * q] = h ? a0 : b0;
            give[i][2 * q + 1] = h ? a1 : b1;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) give[i][k] = __shfl_xor_sync(0xffffffffu, give[i][k], 1);
    const f2 sc = pk(scale, scale);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        f2 X[8], y[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            X[2 * k] = pk(h ? give[2 * q][k] : keep[2 * q][k], h ? give[2 * q + 1][k] : keep[2 * q + 1][k]);
            X[2 * k + 1] = pk(h ? keep[2 * q][k] : give[2 * q][k], h ? keep[2 * q + 1][k] : give[2 * q + 1][k]);
        }
        idct2<8>(X, y);
#pragma unroll
        for (int k = 0; k < 8; ++k) *reinterpret_cast<f2 *>(t + k * 8 + 4 * h + 2 * q) = active ? tc::mul2(y[k], sc) : 0ull;
    }
}

// adds the halves of v to the cells at c0 and c1 (high words; the low words are `low` further on)
__device__ __forceinline__ void box_add(f2 v, int *c0, int *c1, int low)
{
    const f2 hi = fma2(v, pk(kBoxHi, kBoxHi), pk(kBoxRound, kBoxRound));
    const f2 rest = fma2(sub2(hi, pk(kBoxRound, kBoxRound)), pk(-kBoxHiUnit, -kBoxHiUnit), v);
    const f2 lo = fma2(rest, pk(kBoxLo, kBoxLo), pk(kBoxRound, kBoxRound));
    float h0, h1, l0, l1;
    upk(hi, h0, h1);
    upk(lo, l0, l1);
    atomicAdd(c0, __float_as_int(h0) - kBoxRoundBits);
    atomicAdd(c1, __float_as_int(h1) - kBoxRoundBits);
    atomicAdd(c0 + low, __float_as_int(l0) - kBoxRoundBits);
    atomicAdd(c1 + low, __float_as_int(l1) - kBoxRoundBits);
}

// Wiener z stage of one coefficient column (cells t[z * kBT]) of a group of N blocks; returns the sum of the
// squared weights
template <int N>
__device__ __noinline__ float box_wiener(int at, float sg)
{
    extern __shared__ __align__(16) float smem[];
    f2 *t = reinterpret_cast<f2 *>(smem) + at;
    float top = wiener_top(sg);
    const float l2 = wiener_column<N, false>(t, kBT, sg, top);
    return top < kWienerTop ? l2 : wiener_column_exact<N>(t, kBT, sg);
}

// the same for a length without an unrolled transform: the direct sums of both columns at once
__device__ __noinline__ float box_wiener_direct(int at, float sg, int n, const float *fwd, const float *inv)
{
    extern __shared__ __align__(16) float smem[];
    float *t = smem + 2 * at;
    float R[32], X[32];
    direct_sums2<2 * kBT>(t, t + 1, fwd, n, true, R, X);
    float l2 = 0.0f;
    for (int z = 0; z < n; ++z) {
        const float r2 = __fmul_rn(R[z], R[z]);
        const float w = __fdiv_rn(r2, __fadd_rn(r2, sg));
        l2 = __fadd_rn(l2, __fmul_rn(w, w));
        t[2 * kBT * z] = __fmul_rn(X[z], w);
    }
    direct_sums2<2 * kBT>(t, t, inv, n, false, R, X);
    for (int z = 0; z < n; ++z) t[2 * kBT * z] = R[z];
    return l2;
}

template <int G>
__device__ __forceinline__ float box_wiener_any(int at, float sg, int n, const CFArgs &a)
{
    if (n == G) return box_wiener<G>(at, sg);
    if (G > 16 && n == 16) return box_wiener<(G > 16 ? 16 : 1)>(at, sg);
    if (G > 8 && n == 8) return box_wiener<(G > 8 ? 8 : 1)>(at, sg);
    if (n == 4) return box_wiener<4>(at, sg);
    if (n == 2) return box_wiener<2>(at, sg);
    if (n == 1) return box_wiener<1>(at, sg);
    return box_wiener_direct(at, sg, n, dtab_for(a, n, false), dtab_for(a, n, true));
}

// the box, then the slot of block (0, 0), times `unit` (a power of two) to the numerator plane
__device__ __forceinline__ void box_flush(const int *acc, int cells, int slot0, int P, float *num, int ld, int y0, int x0, int bh, int bw,
                                          float unit)
{
    const int qw = bw >> 2;
    for (int e = threadIdx.x; e < bh * qw; e += blockDim.x) {
        const int yy = e / qw, c = 4 * (e - yy * qw);
        const int4 hi = *reinterpret_cast<const int4 *>(acc + yy * P + c), lo = *reinterpret_cast<const int4 *>(acc + cells + yy * P + c);
        float *d = num + (long long)(y0 + yy) * ld + x0 + c;
        if (hi.x | hi.y | hi.z | hi.w | lo.x | lo.y | lo.z | lo.w)
            atomicAdd(reinterpret_cast<float4 *>(d), make_float4(box_value(hi.x, lo.x) * unit, box_value(hi.y, lo.y) * unit,
                                                                 box_value(hi.z, lo.z) * unit, box_value(hi.w, lo.w) * unit));
    }
    if (threadIdx.x < 64) {
        const int e = slot0 + threadIdx.x;
        if (acc[e] | acc[cells + e]) atomicAdd(num + (long long)(threadIdx.x >> 3) * ld + (threadIdx.x & 7), box_value(acc[e], acc[cells + e]) * unit);
    }
}

template <int G, int NP>
__global__ void __launch_bounds__(NP * 64, 8 / NP) cf_box_kernel(CFArgs a, CFBox g)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int GPW = 32 / G;                     // groups per slot
    constexpr int kT = 32 * kBT;                    // cells of a transpose buffer
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5, pair = warp >> 1, role = warp & 1;
    const int p = g.plane[blockIdx.y];
    // tile [bx0, bx1) x [by0, by1) of reference blocks of frame f
    const int rx = blockIdx.x % g.tx, rest = blockIdx.x / g.tx;
    const int rr = rest % g.ty, f = rest / g.ty;
    const int bx0 = (int)((long long)rx * g.nbx / g.tx), bx1 = (int)((long long)(rx + 1) * g.nbx / g.tx);
    const int by0 = (int)((long long)rr * g.nby / g.ty), by1 = (int)((long long)(rr + 1) * g.nby / g.ty);
    const int P = g.pitch;

    // the box: rows [y0, y0 + bh), columns [x0, x0 + bw), whole 16-byte chunks; block (0, 0) in 64 cells after it
    const int y0 = max(0, g.scan_y[by0] - g.range), bh = min(a.H, g.scan_y[by1 - 1] + g.range + 8) - y0;
    const int x0 = max(0, g.scan_x[bx0] - g.range) & ~3;
    const int bw = (min(a.W, g.scan_x[bx1 - 1] + g.range + 8) - x0 + 3) & ~3;
    const int slot0 = g.rows * P, cells = slot0 + 64;
    f2 *tr = reinterpret_cast<f2 *>(smem);
    int *acc = reinterpret_cast<int *>(tr + NP * kT);                  // high words, then low words
    f2 *box = tr + NP * kT + cells;                                             // (reference, source) pairs
    float *red = reinterpret_cast<float *>(box + cells) + pair * 2 * GPW;   // [group of the slot][warp]
    const float *src = a.src[p] + f * a.frame_stride, *ref = a.ref[p] + f * a.frame_stride;
    const int h = lane & 1;
    const int blk = 16 * role + (lane >> 1);        // the lane's block of a slot: group sub, place z
    const int sub = blk / G, z = blk - sub * G;
    // slots run along the tile's rows, GPW groups each
    const int spr = (bx1 - bx0 + GPW - 1) / GPW, nslots = spr * (by1 - by0);
    auto slot_at = [&](int slot, int &bx) -> long long {
        const int sr = slot / spr;
        bx = bx0 + (slot - sr * spr) * GPW;
        return ((long long)f * g.nby + by0 + sr) * g.nbx + bx;
    };
    // length and z-th position of the lane's group of a slot (n = 0: no such group)
    auto fetch = [&](int slot, int &n, uint32_t &pos) {
        n = 0;
        if (slot >= nslots) return;
        int bx;
        const long long grp = slot_at(slot, bx) + sub;
        if (bx + sub < bx1) {
            n = a.count[grp];
            pos = a.pos[grp * G + z];
        }
    };
    int n1 = 0;
    uint32_t pos1 = 0;
    fetch(pair, n1, pos1);
    // all of a thread's loads are in flight together: the staging is one memory latency
    const int qw = bw >> 2, chunks = bh * qw + 16;
    for (int e0 = threadIdx.x; e0 < chunks; e0 += 4 * NP * 64) {
        float4 s4[4], r4[4];
        int at[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int e = e0 + k * NP * 64;
            if (e >= chunks) continue;
            const int yy = e / qw, c = 4 * (e - yy * qw), m = e - (chunks - 16);
            const long long go = m < 0 ? (long long)(y0 + yy) * a.ld + x0 + c : (long long)(m >> 1) * a.ld + 4 * (m & 1);
            at[k] = m < 0 ? yy * P + c : slot0 + 4 * m;
            s4[k] = __ldg(reinterpret_cast<const float4 *>(src + go));
            r4[k] = __ldg(reinterpret_cast<const float4 *>(ref + go));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (e0 + k * NP * 64 >= chunks) continue;
            float4 *d = reinterpret_cast<float4 *>(box + at[k]);
            d[0] = make_float4(r4[k].x, s4[k].x, r4[k].y, s4[k].y);
            d[1] = make_float4(r4[k].z, s4[k].z, r4[k].w, s4[k].w);
        }
    }
    for (int e = threadIdx.x; e < (cells >> 1); e += NP * 64) reinterpret_cast<int4 *>(acc)[e] = make_int4(0, 0, 0, 0);
    __syncthreads();

    f2 *tb = tr + pair * kT + blk * kBT;
    const int sy = lane & 7, sx = lane >> 3;        // the lane's pixel of a block in the scatter (and column sx + 4)
    for (int slot = pair; slot < nslots; slot += NP) {
        const int n = min(n1, G);
        // a place past the group's end filters any block of the box and adds zeros
        const bool active = z < n;
        const int y = unpack_y(pos1), x = unpack_x(pos1);
        const bool in = y >= y0 && y + 8 <= y0 + bh && x >= x0 && x + 8 <= x0 + bw;
        const int off = !active ? 0 : in ? (y - y0) * P + x - x0 : slot0;
        const uint32_t pos = active ? pos1 : 0u;
        fetch(slot + NP, n1, pos1);
        const int bp = off < slot0 ? P : 8;
        const f2 *b = box + off + (h ? 7 * bp : 0);
        const int step = h ? -bp : bp;
        box_forward([&](int i, int c) { return b[i * step + c]; }, tb, h);
        pair_barrier(1 + pair);
        // z stage: warp `role` takes columns 32 role .. 32 role + 31 of every group of the slot
        int sbx;
        const long long sgrp = slot_at(slot, sbx);
#pragma unroll 1
        for (int q = 0; q < GPW; ++q) {
            if (sbx + q >= bx1) break;
            const int nq = min(a.count[sgrp + q], G);
            float l2 = box_wiener_any<G>(pair * kT + q * G * kBT + role * 32 + lane, a.wsig2[p][nq - 1], nq, a);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l2 = __fadd_rn(l2, __shfl_xor_sync(0xffffffffu, l2, o));
            if (lane == 0) red[2 * q + role] = l2;
        }
        pair_barrier(1 + pair);
        const float l2 = __fadd_rn(red[2 * sub], red[2 * sub + 1]);
        const float eps = 1.1920928955078125e-07f;
        const float denW = __fdiv_rn(1.0f, l2 > eps ? l2 : eps);
        box_inverse(reinterpret_cast<float *>(tb), active ? __fdiv_rn(denW, a.amp[n - 1]) : 0.0f, active, h);
        __syncwarp();
        // aggregation, four blocks per step (not unrolled further: the step's code already overflows the
        // instruction caches)
        const float *v = reinterpret_cast<const float *>(tr + pair * kT + 16 * role * kBT) + lane;
        int *cell = acc + sy * P + sx, *cell0 = acc + sy * 8 + sx;
#pragma unroll 1
        for (int i = 0; i < 16; i += 4) {
            f2 e[4];
            int o[4];
            bool fits = true;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                o[k] = __shfl_sync(0xffffffffu, off, 2 * (i + k));
                const float e0 = v[(i + k) * 2 * kBT], e1 = v[(i + k) * 2 * kBT + 32];
                fits = fits && fabsf(e0) < kBoxMax && fabsf(e1) < kBoxMax;
                e[k] = pk(e0, e1);
            }
            if (__all_sync(0xffffffffu, fits)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int *c = (o[k] < slot0 ? cell : cell0) + o[k];
                    box_add(e[k], c, c + 4, cells);
                }
            } else {
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    const uint32_t pi = __shfl_sync(0xffffffffu, pos, 2 * (i + k));
                    float *np = a.num[p] + f * a.frame_stride + (long long)(unpack_y(pi) + sy) * a.ld + unpack_x(pi) + sx;
                    atomicAdd(np, v[(i + k) * 2 * kBT]);
                    atomicAdd(np + 4, v[(i + k) * 2 * kBT + 32]);
                }
            }
        }
        if (active && h == 0) atomicAdd(a.wmap[p] + f * a.frame_stride + (long long)unpack_y(pos) * a.ld + unpack_x(pos), denW);
        __syncwarp();
    }

    __syncthreads();
    box_flush(acc, cells, slot0, P, a.num[p] + f * a.frame_stride, a.ld, y0, x0, bh, bw, 1.0f);
}

// ---- Basic: hard threshold ------------------------------------------------------------------------------
// A pair of warps takes two slots at once, packed: the halves of every cell and register are the blocks at
// the same place of slots A and B, through both directions of the transform.
// Bound: the shared-memory pipe (random-row loads of the blocks, transposes, and four native atomics a
// pixel pair: 6.7 k of a step's 25 k clocks are atomics).  1920x1080 RGB x 8, step 4, G = 16: 12.6 ms with
// per-lane gathers and float atomics on the plane (cf_fast_kernel), 8.6 ms now (8.3 ms on an absolute grid).

// A term is a pixel over its group's kept count, so its size follows the clip's, and an absolute grid would keep
// fewer bits of a clip of small values than fp32 sums do.  So
// - a tile whose largest staged magnitude is below kTileMin is filtered in units that put it in [32, 64), a power
//   of two: its terms are those of the clip, scaled;
// - a group whose terms are still below kBoxMin (a dark part of a bright tile) goes to the plane directly, as
//   blocks of large terms do.
// The grid's rounding is then at most 2^-19 of the largest term of the group's first block (of its seventeenth for the
// second warp of a group of 32), and usually far less: the test takes one coefficient's share of it.  A pixel
// averages the roundings of dozens of terms.
constexpr float kTileMin = 0.0625f;                                            // 2^-4
constexpr float kBoxMin = 6.103515625e-5f;                                     // 2^-14

__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

// bits of a tile's scale, from the bits of its largest magnitude; limited so that neither the scale nor its inverse
// underflows
__device__ __forceinline__ unsigned box_scale_bits(unsigned top)
{
    return top < __float_as_uint(kTileMin) ? (unsigned)min(259 - (int)(top >> 23), 253) << 23 : 127u << 23;
}

// the block of slot A (low halves) and of slot B at a place, one of which may not go to the box: each to the cells
// (at ca, cb, and 4 further on for the second pixel) or to the plane (at na, nb) times `down`
__device__ __noinline__ void box_add_apart(f2 e0, f2 e1, int *ca, int *cb, int low, float *na, float *nb, float down, bool apartA, bool apartB)
{
    float a0, b0, a1, b1;
    upk(e0, a0, b0);
    upk(e1, a1, b1);
    const bool fa = !apartA && __all_sync(0xffffffffu, fabsf(a0) < kBoxMax && fabsf(a1) < kBoxMax);
    const bool fb = !apartB && __all_sync(0xffffffffu, fabsf(b0) < kBoxMax && fabsf(b1) < kBoxMax);
    if (fa || fb) {
        box_add(pk(fa ? a0 : 0.0f, fb ? b0 : 0.0f), ca, cb, low);
        box_add(pk(fa ? a1 : 0.0f, fb ? b1 : 0.0f), ca + 4, cb + 4, low);
    }
    if (!fa) {
        atomicAdd(na, a0 * down);
        atomicAdd(na + 4, a1 * down);
    }
    if (!fb) {
        atomicAdd(nb, b0 * down);
        atomicAdd(nb + 4, b1 * down);
    }
}

// hard threshold of both halves of x, counted in the halves of kept
__device__ __forceinline__ f2 keep2(f2 x, float ta, float tb, int &kept)
{
    float a, b;
    upk(x, a, b);
    const bool ka = fabsf(a) > ta, kb = fabsf(b) > tb;
    kept += (ka ? 1 : 0) + (kb ? 1 << 16 : 0);
    return pk(ka ? a : 0.0f, kb ? b : 0.0f);
}

// z stage of one coefficient column of two groups of N blocks; thresholds t0 (z = 0) and t1; returns the
// kept counts in the halves of an int
template <int N>
__device__ __noinline__ int box_hard(int at, float t0, float t1)
{
    extern __shared__ __align__(16) float smem[];
    f2 *t = reinterpret_cast<f2 *>(smem) + at;
    f2 x[N], X[N], y[N];
#pragma unroll
    for (int z = 0; z < N; ++z) x[z] = t[z * kBT];
    int kept = 0;
    fdct2<N>(x, [&](int k, int st, const auto &v) {
#pragma unroll
        for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) {
            const float th = k + i * st == 0 ? t0 : t1;
            X[k + i * st] = keep2(v[i], th, th, kept);
        }
    });
    if constexpr (N == 1) y[0] = X[0];
    else idct2<N>(X, y);
#pragma unroll
    for (int z = 0; z < N; ++z) t[z * kBT] = y[z];
    return kept;
}

// the same for one of the two groups alone (t: its half of the column), any length
template <int N>
__device__ __forceinline__ int box_hard_half(float *t, float t0, float t1)
{
    float x[N], X[N];
#pragma unroll
    for (int z = 0; z < N; ++z) x[z] = t[2 * z * kBT];
    fdct_reg<N>(x, X);
    int kept = 0;
#pragma unroll
    for (int z = 0; z < N; ++z) {
        const bool k = fabsf(X[z]) > (z ? t1 : t0);
        kept += k;
        X[z] = k ? X[z] : 0.0f;
    }
    idct_reg<N>(X, x);
#pragma unroll
    for (int z = 0; z < N; ++z) t[2 * z * kBT] = x[z];
    return kept;
}

__device__ __noinline__ int box_hard_any(int at, int half, float t0, float t1, int n, const float *fwd, const float *inv)
{
    extern __shared__ __align__(16) float smem[];
    float *t = smem + 2 * at + half;
    switch (n) {
    case 0: return 0;
    case 1: return box_hard_half<1>(t, t0, t1);
    case 2: return box_hard_half<2>(t, t0, t1);
    case 4: return box_hard_half<4>(t, t0, t1);
    case 8: return box_hard_half<8>(t, t0, t1);
    case 16: return box_hard_half<16>(t, t0, t1);
    case 32: return box_hard_half<32>(t, t0, t1);
    }
    float X[32], Y[32];
    direct_sums2<2 * kBT>(t, t, fwd, n, true, X, Y);
    int kept = 0;
    for (int z = 0; z < n; ++z) {
        const bool k = fabsf(X[z]) > (z ? t1 : t0);
        kept += k;
        t[2 * z * kBT] = k ? X[z] : 0.0f;
    }
    direct_sums2<2 * kBT>(t, t, inv, n, false, X, Y);
    for (int z = 0; z < n; ++z) t[2 * z * kBT] = X[z];
    return kept;
}

// z stage of the two groups at a column, of ma and mb blocks (0: no group): the warp's kept counts in the halves
// of an int.  Groups of the same full length go together, others one by one.
template <int G>
__device__ __forceinline__ int box_hard_pair(int at, const CFArgs &a, int p, int fxy, int ma, int mb)
{
    int kept = 0;
    if (ma == G && mb == G) kept = box_hard<G>(at, a.thr4[p][G - 1][fxy + 1], a.thr4[p][G - 1][fxy]);
    else {
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            const int m = half ? mb : ma, i = max(m, 1) - 1;
            kept += box_hard_any(at, half, a.thr4[p][i][fxy + 1], a.thr4[p][i][fxy], m, dtab_for(a, m, false),
                                 dtab_for(a, m, true)) << (16 * half);
        }
    }
    return __reduce_add_sync(0xffffffffu, kept);
}

// Inverse 2-D transform of both halves of the cells at `t`, scaled, in place: pixel (y, x) to cell 8 x + y.
// Lane half h inverts the columns 2k + h, then the rows 2i + h.
__device__ __forceinline__ void box_inverse2(f2 *t, f2 scale, bool activeA, bool activeB, int h)
{
    f2 keep[4][4], give[4][4];            // [row][column]
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        f2 X[8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) X[i] = t[i * 8 + 2 * k + h];
        idct2<8>(X, y);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            keep[i][k] = h ? y[2 * i + 1] : y[2 * i];
            give[i][k] = h ? y[2 * i] : y[2 * i + 1];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) give[i][k] = shfl_pair(give[i][k]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f2 X[8], y[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            X[2 * k] = h ? give[i][k] : keep[i][k];
            X[2 * k + 1] = h ? keep[i][k] : give[i][k];
        }
        idct2<8>(X, y);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float a, b;
            upk(tc::mul2(y[k], scale), a, b);
            t[k * 8 + 2 * i + h] = pk(activeA ? a : 0.0f, activeB ? b : 0.0f);
        }
    }
}

template <int G, int NP>
__global__ void __launch_bounds__(NP * 64, 8 / NP) cf_boxh_kernel(CFArgs a, CFBox g)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int GPW = 32 / G;                     // groups per slot
    constexpr int kT = 32 * kBT;                    // cells of a transpose buffer
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5, pair = warp >> 1, role = warp & 1;
    const int p = g.plane[blockIdx.y];
    const int rx = blockIdx.x % g.tx, rest = blockIdx.x / g.tx;
    const int rr = rest % g.ty, f = rest / g.ty;
    const int bx0 = (int)((long long)rx * g.nbx / g.tx), bx1 = (int)((long long)(rx + 1) * g.nbx / g.tx);
    const int by0 = (int)((long long)rr * g.nby / g.ty), by1 = (int)((long long)(rr + 1) * g.nby / g.ty);
    const int P = g.pitch;
    const int y0 = max(0, g.scan_y[by0] - g.range), bh = min(a.H, g.scan_y[by1 - 1] + g.range + 8) - y0;
    const int x0 = max(0, g.scan_x[bx0] - g.range) & ~3;
    const int bw = (min(a.W, g.scan_x[bx1 - 1] + g.range + 8) - x0 + 3) & ~3;
    const int slot0 = g.rows * P, cells = slot0 + 64;
    f2 *tr = reinterpret_cast<f2 *>(smem);
    int *acc = reinterpret_cast<int *>(tr + NP * kT);                  // high words, then low words
    float *box = reinterpret_cast<float *>(acc + 2 * cells);
    unsigned *tops = reinterpret_cast<unsigned *>(box + cells);        // [warp]
    int *red = reinterpret_cast<int *>(tops + 2 * NP) + pair * 2 * GPW;  // [group of the slots][warp]
    const float *src = a.src[p] + f * a.frame_stride;
    const int h = lane & 1;
    const int blk = 16 * role + (lane >> 1);        // the lane's block of a slot: group sub, place z
    const int sub = blk / G, z = blk - sub * G;
    const int spr = (bx1 - bx0 + GPW - 1) / GPW, nslots = spr * (by1 - by0);
    // first group of a slot, and how many groups it has
    auto slot_at = [&](int slot, int &groups) -> long long {
        const int sr = slot / spr, bx = bx0 + (slot - sr * spr) * GPW;
        groups = slot < nslots ? min(GPW, bx1 - bx) : 0;
        return ((long long)f * g.nby + by0 + sr) * g.nbx + bx;
    };
    auto fetch = [&](int slot, int &n, uint32_t &pos) {
        int groups;
        const long long grp = slot_at(slot, groups) + sub;
        n = 0;
        if (sub < groups) {
            n = a.count[grp];
            pos = a.pos[grp * G + z];
        }
    };
    int nA = 0, nB = 0;
    uint32_t pA = 0, pB = 0;
    fetch(2 * pair, nA, pA);
    fetch(2 * pair + 1, nB, pB);
    const int qw = bw >> 2, chunks = bh * qw + 16;
    for (int e = threadIdx.x; e < chunks; e += NP * 64) {
        const int yy = e / qw, c = 4 * (e - yy * qw), m = e - (chunks - 16);
        if (m < 0) tc::cp_async16(box + yy * P + c, src + (long long)(y0 + yy) * a.ld + x0 + c);
        else tc::cp_async16(box + slot0 + 4 * m, src + (long long)(m >> 1) * a.ld + 4 * (m & 1));
    }
    for (int e = threadIdx.x; e < (cells >> 1); e += NP * 64) reinterpret_cast<int4 *>(acc)[e] = make_int4(0, 0, 0, 0);
    tc::cp_async_wait_all();
    // largest finite magnitude of the plane's pixels among the thread's own copies, then of the tile
    unsigned top = 0u;
    for (int e = threadIdx.x; e < chunks; e += NP * 64) {
        const int yy = e / qw, c = 4 * (e - yy * qw), m = e - (chunks - 16);
        const float4 v = *reinterpret_cast<const float4 *>(box + (m < 0 ? yy * P + c : slot0 + 4 * m));
        const unsigned u[4] = {abs_bits(v.x), abs_bits(v.y), abs_bits(v.z), abs_bits(v.w)};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (u[k] < 0x7f800000u && (m >= 0 || x0 + c + k < a.W)) top = max(top, u[k]);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) tops[warp] = top;
    __syncthreads();
    const unsigned sb = box_scale_bits(__reduce_max_sync(0xffffffffu, tops[lane & (2 * NP - 1)]));
    const float up = __uint_as_float(sb), down = __uint_as_float((254u << 23) - sb);

    f2 *tb = tr + pair * kT + blk * kBT;
    const int sy = lane & 7, sx = lane >> 3;        // the lane's pixel of a block in the scatter (and column sx + 4)
    auto place = [&](int n, uint32_t pos) {
        const int y = unpack_y(pos), x = unpack_x(pos);
        const bool in = y >= y0 && y + 8 <= y0 + bh && x >= x0 && x + 8 <= x0 + bw;
        return z >= n ? 0 : in ? (y - y0) * P + x - x0 : slot0;
    };
    for (int slot = 2 * pair; slot < nslots; slot += 2 * NP) {
        const int na = min(nA, G), nb = min(nB, G);
        const bool actA = z < na, actB = z < nb;
        const uint32_t posA = actA ? pA : 0u, posB = actB ? pB : 0u;
        const int offA = place(na, posA), offB = place(nb, posB);
        fetch(slot + 2 * NP, nA, pA);
        fetch(slot + 2 * NP + 1, nB, pB);
        {
            const int ba = offA < slot0 ? P : 8, bb = offB < slot0 ? P : 8;
            const float *ca = box + offA + (h ? 7 * ba : 0), *cb = box + offB + (h ? 7 * bb : 0);
            const int sa = h ? -ba : ba, sb = h ? -bb : bb;
            box_forward([&](int i, int c) { return pk(ca[i * sa + c], cb[i * sb + c]); }, tb, h);
        }
        pair_barrier(1 + pair);
        int gA, gB;
        const long long grpA = slot_at(slot, gA), grpB = slot_at(slot + 1, gB);
        const int col = role * 32 + lane, fxy = ((col & 7) == 0) + ((col >> 3) == 0);
#pragma unroll 1
        for (int q = 0; q < GPW; ++q) {
            const int ma = q < gA ? min(a.count[grpA + q], G) : 0, mb = q < gB ? min(a.count[grpB + q], G) : 0;
            const int at = pair * kT + q * G * kBT + col;
            const int kept = box_hard_pair<G>(at, a, p, fxy, ma, mb);
            if (lane == 0) red[2 * q + role] = kept;
        }
        pair_barrier(1 + pair);
        const int kept = red[2 * sub] + red[2 * sub + 1], kA = kept & 0xffff, kB = kept >> 16;
        if (a.retained && z == 0 && h == 0) {
            if (sub < gA) a.retained[(long long)p * a.ngroups + grpA + sub] = kA;
            if (sub < gB) a.retained[(long long)p * a.ngroups + grpB + sub] = kB;
        }
        const float dA = kA < 1 ? 1.0f : __fdiv_rn(1.0f, (float)kA), dB = kB < 1 ? 1.0f : __fdiv_rn(1.0f, (float)kB);
        const float wA = actA ? __fdiv_rn(dA, a.amp[na - 1]) * up : 0.0f, wB = actB ? __fdiv_rn(dB, a.amp[nb - 1]) * up : 0.0f;
        // largest coefficient of the first of the warp's blocks of the lane's group, by the lanes of that group
        constexpr int kLanes = G < 16 ? 2 * G : 32;
        unsigned ta = 0u, tb0 = 0u;
#pragma unroll
        for (int j = lane & (kLanes - 1); j < 64; j += kLanes) {
            float u, w;
            upk(tr[pair * kT + (16 * role + (lane & ~(kLanes - 1)) / 2) * kBT + j], u, w);
            ta = max(ta, abs_bits(u));
            tb0 = max(tb0, abs_bits(w));
        }
        __syncwarp();
        box_inverse2(tb, pk(wA, wB), actA, actB, h);
        __syncwarp();
        if constexpr (kLanes == 32) {
            ta = __reduce_max_sync(0xffffffffu, ta);
            tb0 = __reduce_max_sync(0xffffffffu, tb0);
        } else {
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) {
                ta = max(ta, __shfl_xor_sync(0xffffffffu, ta, o));
                tb0 = max(tb0, __shfl_xor_sync(0xffffffffu, tb0, o));
            }
        }
        // a pixel is, on the mean square, at least as large as any one of its block's coefficients
        const float tA = __uint_as_float(ta) * wA, tB = __uint_as_float(tb0) * wB;
        const bool apartA = actA && tA > 0.0f && tA < kBoxMin, apartB = actB && tB > 0.0f && tB < kBoxMin;
        const unsigned apart = __ballot_sync(0xffffffffu, apartA || apartB), places = __ballot_sync(0xffffffffu, actA || actB);
        // aggregation, four blocks (two places of both slots) per step
        const f2 *v = tr + pair * kT + 16 * role * kBT + lane;
        int *cell = acc + sy * P + sx, *cell0 = acc + sy * 8 + sx;
        unsigned later = 0u;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            f2 e[4];
            int oa[2], ob[2];
            bool fits = true;
            if (!(places >> 2 * i & 15u)) continue;     // past the groups' ends
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                oa[k] = __shfl_sync(0xffffffffu, offA, 2 * (i + k));
                ob[k] = __shfl_sync(0xffffffffu, offB, 2 * (i + k));
                e[2 * k] = v[(i + k) * kBT];
                e[2 * k + 1] = v[(i + k) * kBT + 32];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float u, w;
                upk(e[k], u, w);
                fits = fits && fabsf(u) < kBoxMax && fabsf(w) < kBoxMax;
            }
            if (!apart && __all_sync(0xffffffffu, fits)) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    int *ca = (oa[k] < slot0 ? cell : cell0) + oa[k], *cb = (ob[k] < slot0 ? cell : cell0) + ob[k];
                    box_add(e[2 * k], ca, cb, cells);
                    box_add(e[2 * k + 1], ca + 4, cb + 4, cells);
                }
            } else {
                later |= 3u << i;
            }
        }
        // places with a block that the box does not take: each block to its own destination
        for (; later; later &= later - 1) {
            const int i = __ffs(later) - 1;
            const int ia = __shfl_sync(0xffffffffu, offA, 2 * i), ib = __shfl_sync(0xffffffffu, offB, 2 * i);
            const uint32_t qa = __shfl_sync(0xffffffffu, posA, 2 * i), qb = __shfl_sync(0xffffffffu, posB, 2 * i);
            float *num = a.num[p] + f * a.frame_stride + (long long)sy * a.ld + sx;
            box_add_apart(v[i * kBT], v[i * kBT + 32], (ia < slot0 ? cell : cell0) + ia, (ib < slot0 ? cell : cell0) + ib, cells,
                          num + (long long)unpack_y(qa) * a.ld + unpack_x(qa), num + (long long)unpack_y(qb) * a.ld + unpack_x(qb), down,
                          __shfl_sync(0xffffffffu, apartA, 2 * i), __shfl_sync(0xffffffffu, apartB, 2 * i));
        }
        if (h == 0) {
            float *wm = a.wmap[p] + f * a.frame_stride;
            if (actA) atomicAdd(wm + (long long)unpack_y(posA) * a.ld + unpack_x(posA), dA);
            if (actB) atomicAdd(wm + (long long)unpack_y(posB) * a.ld + unpack_x(posB), dB);
        }
        __syncwarp();
    }

    __syncthreads();
    box_flush(acc, cells, slot0, P, a.num[p] + f * a.frame_stride, a.ld, y0, x0, bh, bw, down);
}

// ---- the same warp pairs without a box --------------------------------------------------------------------
// V-BM3D, whose groups' blocks lie in up to 2 radius + 1 frames, and search windows whose box holds too few groups:
// blocks are read from and added to the planes one per warp step (lane = row and column of half a block), through
// the transpose buffer.
// Bound: latency of the steps and the L2's atomics.  1280x720 YUV x 7, radius 3, Final, G = 8: 7.4 ms
// with per-lane gathers and atomics (cf_fast_kernel), 4.8 ms here.

// offsets of the lane's block in the source planes and in the accumulators (locate() with 64-bit offsets)
__device__ __forceinline__ void pair_locate(const CFArgs &a, long long grp, uint32_t pk, long long &src, long long &acc)
{
    const long long f = grp / a.blocks_per_frame;
    if (!a.vbm3d) {
        src = acc = f * a.frame_stride + (long long)unpack_y(pk) * a.ld + unpack_x(pk);
    } else {
        const int z = unpack3_z(pk);
        const long long at = (long long)unpack3_y(pk) * a.ld + unpack3_x(pk);
        src = ((long long)a.win_base[f] + z) * a.frame_stride + at;
        acc = (f * a.slots + a.slot0[f] + z) * a.acc_stride + at;
    }
}

template <int G, int NP>
__global__ void __launch_bounds__(NP * 64, 8 / NP) cf_pair_kernel(const __grid_constant__ CFArgs a)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int GPW = 32 / G, kT = 32 * kBT;
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5, pair = warp >> 1, role = warp & 1;
    f2 *tr = reinterpret_cast<f2 *>(smem) + pair * kT;
    float *red = smem + 2 * NP * kT + pair * 2 * GPW;
    const int h = lane & 1, blk = 16 * role + (lane >> 1), sub = blk / G, z = blk - sub * G;
    f2 *tb = tr + blk * kBT, *tw = tr + 16 * role * kBT;
    const int ry = lane >> 3, cx = lane & 7;
    const long long nslots = (a.ngroups + GPW - 1) / GPW;
    for (long long slot = (long long)blockIdx.x * NP + pair; slot < nslots; slot += (long long)gridDim.x * NP) {
        const long long grp = slot * GPW + sub;
        const int n = grp < a.ngroups ? min(a.count[grp], G) : 0;
        const bool active = z < n;
        long long so = 0, ao = 0;
        if (active) pair_locate(a, grp, a.pos[grp * G + z], so, ao);
        for (int p = 0; p < 3; ++p) {
            if (!a.process[p]) continue;
            const float *src = a.src[p], *ref = a.ref[p];
            __syncwarp();
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
                const long long o = __shfl_sync(0xffffffffu, so, 2 * i) + (long long)ry * a.ld + cx;
                tw[i * kBT + lane] = pk(__ldg(ref + o), __ldg(src + o));
                tw[i * kBT + 32 + lane] = pk(__ldg(ref + o + 4ll * a.ld), __ldg(src + o + 4ll * a.ld));
            }
            __syncwarp();
            {
                f2 x[4][8];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[i][k] = tb[(h ? 7 - i : i) * 8 + k];
                __syncwarp();
                box_forward([&](int i, int k) { return x[i][k]; }, tb, h);
            }
            pair_barrier(1 + pair);
#pragma unroll 1
            for (int q = 0; q < GPW; ++q) {
                if (slot * GPW + q >= a.ngroups) break;
                const int nq = min(a.count[slot * GPW + q], G);
                float l2 = box_wiener_any<G>(pair * kT + q * G * kBT + role * 32 + lane, a.wsig2[p][nq - 1], nq, a);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) l2 = __fadd_rn(l2, __shfl_xor_sync(0xffffffffu, l2, o));
                if (lane == 0) red[2 * q + role] = l2;
            }
            pair_barrier(1 + pair);
            const float l2 = __fadd_rn(red[2 * sub], red[2 * sub + 1]);
            const float eps = 1.1920928955078125e-07f;
            const float denW = __fdiv_rn(1.0f, l2 > eps ? l2 : eps);
            box_inverse(reinterpret_cast<float *>(tb), active ? __fdiv_rn(denW, a.amp[n - 1]) : 0.0f, active, h);
            __syncwarp();
            const unsigned mask = __ballot_sync(0xffffffffu, active);
            float *num = a.num[p];
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
                const long long o = __shfl_sync(0xffffffffu, ao, 2 * i) + (long long)ry * a.ld + cx;
                const float *v = reinterpret_cast<const float *>(tw + i * kBT) + cx * 8 + ry;
                if (mask >> (2 * i) & 1) {
                    atomicAdd(num + o, v[0]);
                    atomicAdd(num + o + 4ll * a.ld, v[4]);
                }
            }
            if (active && h == 0) atomicAdd(a.wmap[p] + ao, denW);
        }
    }
}

template <int G, int NP>
__global__ void __launch_bounds__(NP * 64, 8 / NP) cf_pairh_kernel(const __grid_constant__ CFArgs a)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int GPW = 32 / G, kT = 32 * kBT;
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5, pair = warp >> 1, role = warp & 1;
    f2 *tr = reinterpret_cast<f2 *>(smem) + pair * kT;
    int *red = reinterpret_cast<int *>(smem + 2 * NP * kT) + pair * 2 * GPW;
    const int h = lane & 1, blk = 16 * role + (lane >> 1), sub = blk / G, z = blk - sub * G;
    f2 *tb = tr + blk * kBT, *tw = tr + 16 * role * kBT;
    const int ry = lane >> 3, cx = lane & 7;
    const int col = role * 32 + lane, fxy = ((col & 7) == 0) + ((col >> 3) == 0);
    const long long nslots = (a.ngroups + GPW - 1) / GPW;
    for (long long slot = 2 * ((long long)blockIdx.x * NP + pair); slot < nslots; slot += 2ll * gridDim.x * NP) {
        const long long gA = slot * GPW + sub, gB = gA + GPW;
        const int na = gA < a.ngroups ? min(a.count[gA], G) : 0, nb = gB < a.ngroups ? min(a.count[gB], G) : 0;
        const bool actA = z < na, actB = z < nb;
        long long sA = 0, oA = 0, sB = 0, oB = 0;
        if (actA) pair_locate(a, gA, a.pos[gA * G + z], sA, oA);
        if (actB) pair_locate(a, gB, a.pos[gB * G + z], sB, oB);
        for (int p = 0; p < 3; ++p) {
            if (!a.process[p]) continue;
            const float *src = a.src[p];
            __syncwarp();
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
                const long long u = __shfl_sync(0xffffffffu, sA, 2 * i) + (long long)ry * a.ld + cx;
                const long long v = __shfl_sync(0xffffffffu, sB, 2 * i) + (long long)ry * a.ld + cx;
                tw[i * kBT + lane] = pk(__ldg(src + u), __ldg(src + v));
                tw[i * kBT + 32 + lane] = pk(__ldg(src + u + 4ll * a.ld), __ldg(src + v + 4ll * a.ld));
            }
            __syncwarp();
            {
                f2 x[4][8];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[i][k] = tb[(h ? 7 - i : i) * 8 + k];
                __syncwarp();
                box_forward([&](int i, int k) { return x[i][k]; }, tb, h);
            }
            pair_barrier(1 + pair);
#pragma unroll 1
            for (int q = 0; q < GPW; ++q) {
                const long long ga = slot * GPW + q, gb = ga + GPW;
                const int ma = ga < a.ngroups ? min(a.count[ga], G) : 0, mb = gb < a.ngroups ? min(a.count[gb], G) : 0;
                const int kept = box_hard_pair<G>(pair * kT + q * G * kBT + col, a, p, fxy, ma, mb);
                if (lane == 0) red[2 * q + role] = kept;
            }
            pair_barrier(1 + pair);
            const int kept = red[2 * sub] + red[2 * sub + 1], kA = kept & 0xffff, kB = kept >> 16;
            if (a.retained && z == 0 && h == 0) {
                if (na) a.retained[(long long)p * a.ngroups + gA] = kA;
                if (nb) a.retained[(long long)p * a.ngroups + gB] = kB;
            }
            const float dA = kA < 1 ? 1.0f : __fdiv_rn(1.0f, (float)kA), dB = kB < 1 ? 1.0f : __fdiv_rn(1.0f, (float)kB);
            box_inverse2(tb, pk(actA ? __fdiv_rn(dA, a.amp[na - 1]) : 0.0f, actB ? __fdiv_rn(dB, a.amp[nb - 1]) : 0.0f), actA, actB, h);
            __syncwarp();
            const unsigned mA = __ballot_sync(0xffffffffu, actA), mB = __ballot_sync(0xffffffffu, actB);
            float *num = a.num[p];
#pragma unroll 4
            for (int i = 0; i < 16; ++i) {
                const long long u = __shfl_sync(0xffffffffu, oA, 2 * i) + (long long)ry * a.ld + cx;
                const long long v = __shfl_sync(0xffffffffu, oB, 2 * i) + (long long)ry * a.ld + cx;
                const f2 *e = tw + i * kBT + cx * 8 + ry;
                float a0, b0, a1, b1;
                upk(e[0], a0, b0);
                upk(e[4], a1, b1);
                if (mA >> (2 * i) & 1) {
                    atomicAdd(num + u, a0);
                    atomicAdd(num + u + 4ll * a.ld, a1);
                }
                if (mB >> (2 * i) & 1) {
                    atomicAdd(num + v, b0);
                    atomicAdd(num + v + 4ll * a.ld, b1);
                }
            }
            if (h == 0) {
                if (actA) atomicAdd(a.wmap[p] + oA, dA);
                if (actB) atomicAdd(a.wmap[p] + oB, dB);
            }
        }
    }
}

}  // namespace bm3d
