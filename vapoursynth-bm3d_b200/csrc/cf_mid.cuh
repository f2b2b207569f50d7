// cf_mid.cuh -- K3+K4, plain form: the collaborative filter of groups of at most 32 blocks of 2 x 2 to
// 16 x 16 pixels that are not the 8 x 8 blocks of the box form (profile "vn" refines with 11 x 11 ones).
//
// One CTA of four warps per group, the group in shared memory: every 1-D transform is one thread's, a row,
// a column or a coefficient column along z.  Power-of-two lengths use the unrolled butterflies of common.cuh,
// others the direct sums over a table in shared memory, all outputs of a row side by side (one pixel read and
// the table's row, the same for every lane, per step).  The Wiener filter holds (reference, source) pairs and
// transforms both at once with packed arithmetic.  Same operations in the same order as cf_generic_kernel.
// Bound: FP32 multiply-adds of the direct sums (121 per 11-point transform).  cf_generic_kernel keeps one
// group per warp in global scratch, a transform's inputs in local memory; 1280x720 gray, 11 x 11 blocks,
// groups of 32: 7.3 ms there, 1.20 ms here.
#pragma once

#include "cf_box.cuh"

namespace bm3d {

constexpr int kMidThreads = 128;

// arithmetic on a cell: a float (Basic) or a (reference, source) pair (Final)
__device__ __forceinline__ float cell_mul(float a, float c) { return __fmul_rn(a, c); }
__device__ __forceinline__ float cell_fma(float a, float c, float s) { return __fmaf_rn(a, c, s); }
__device__ __forceinline__ f2 cell_mul(f2 a, float c) { return tc::mul2(a, pk(c, c)); }
__device__ __forceinline__ f2 cell_fma(f2 a, float c, f2 s) { return fma2(a, pk(c, c), s); }

template <int N>
__device__ __forceinline__ void cell_fdct(const float (&x)[N], float (&X)[N]) { fdct_reg<N>(x, X); }
template <int N>
__device__ __forceinline__ void cell_fdct(const f2 (&x)[N], f2 (&X)[N])
{
    fdct2<N>(x, [&](int k, int st, const auto &v) {
#pragma unroll
        for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) X[k + i * st] = v[i];
    });
}

// One transform of length B (BM: B rounded up, or B itself for a power of two) at v with the given stride of
// cells, in place.  tab: rows j = 0 .. B - 1 of BM coefficients t[k][j] (zero past B).
template <int BM, bool DIRECT, bool INVERSE, class T>
__device__ __forceinline__ void mid_transform(T *v, int stride, int B, const float *tab)
{
    if constexpr (!DIRECT) {
        T x[BM], X[BM];
#pragma unroll
        for (int k = 0; k < BM; ++k) x[k] = v[k * stride];
        if constexpr (INVERSE) idct_reg<BM>(x, X);
        else cell_fdct<BM>(x, X);
#pragma unroll
        for (int k = 0; k < BM; ++k) v[k * stride] = X[k];
    } else {
        T acc[BM];
        const T x0 = v[0];
#pragma unroll
        for (int k = 0; k < BM; k += 4) {
            const float4 c = *reinterpret_cast<const float4 *>(tab + k);
            // the inverse's first term is X_0 itself (its coefficients are ones)
            acc[k] = INVERSE ? x0 : cell_mul(x0, c.x);
            acc[k + 1] = INVERSE ? x0 : cell_mul(x0, c.y);
            acc[k + 2] = INVERSE ? x0 : cell_mul(x0, c.z);
            acc[k + 3] = INVERSE ? x0 : cell_mul(x0, c.w);
        }
#pragma unroll 1
        for (int j = 1; j < B; ++j) {
            const T x = v[j * stride];
#pragma unroll
            for (int k = 0; k < BM; k += 4) {
                const float4 c = *reinterpret_cast<const float4 *>(tab + j * BM + k);
                acc[k] = cell_fma(x, c.x, acc[k]);
                acc[k + 1] = cell_fma(x, c.y, acc[k + 1]);
                acc[k + 2] = cell_fma(x, c.z, acc[k + 2]);
                acc[k + 3] = cell_fma(x, c.w, acc[k + 3]);
            }
        }
#pragma unroll
        for (int k = 0; k < BM; ++k)
            if (k < B) v[k * stride] = acc[k];
    }
}

// z stage of a column of n cells at v: transform, shrinkage, inverse; the filtered source in the float at v (the
// pairs' low word), kept count or sum of squared weights returned
template <int N>
__device__ __forceinline__ float mid_z(f2 *v, int stride, float sg, float)
{
    float top = wiener_top(sg);
    const float l2 = wiener_column<N, false>(v, stride, sg, top);
    return top < kWienerTop ? l2 : wiener_column_exact<N>(v, stride, sg);
}

template <int N>
__device__ __forceinline__ float mid_z(float *v, int stride, float t0, float t1)
{
    float x[N], X[N];
    int kept = 0;
#pragma unroll
    for (int z = 0; z < N; ++z) x[z] = v[z * stride];
    fdct_reg<N>(x, X);
#pragma unroll
    for (int z = 0; z < N; ++z) {
        const bool k = fabsf(X[z]) > (z ? t1 : t0);
        kept += k;
        X[z] = k ? X[z] : 0.0f;
    }
    idct_reg<N>(X, x);
#pragma unroll
    for (int z = 0; z < N; ++z) v[z * stride] = x[z];
    return (float)kept;
}

// out[k] = sum_j t[k][j] x[j] for a column of floats at v (stride in floats), any length up to 32
__device__ __forceinline__ void mid_direct(const float *v, int stride, const float *t, int n, bool inverse, float *out)
{
    for (int k0 = 0; k0 < n; k0 += kDirectChains) {
        float a[kDirectChains];
        const float x0 = v[0];
#pragma unroll
        for (int i = 0; i < kDirectChains; ++i) a[i] = inverse ? x0 : __fmul_rn(x0, __ldg(t + min(k0 + i, n - 1) * n));
        for (int j = 1; j < n; ++j) {
            const float x = v[j * stride];
#pragma unroll
            for (int i = 0; i < kDirectChains; ++i) a[i] = __fmaf_rn(x, __ldg(t + min(k0 + i, n - 1) * n + j), a[i]);
        }
#pragma unroll
        for (int i = 0; i < kDirectChains; ++i)
            if (k0 + i < n) out[k0 + i] = a[i];
    }
}

template <class T>
__device__ __noinline__ float mid_z_direct(T *v, int stride, float p0, float p1, int n, const float *fwd, const float *inv)
{
    constexpr bool W = sizeof(T) == 8;
    float *t = reinterpret_cast<float *>(v);
    const int fs = W ? 2 * stride : stride;
    float X[32], r = 0.0f;
    if constexpr (W) {
        float S[32];
        mid_direct(t + 1, fs, fwd, n, false, S);
        mid_direct(t, fs, fwd, n, false, X);
        for (int z = 0; z < n; ++z) {
            const float r2 = __fmul_rn(X[z], X[z]);
            const float w = __fdiv_rn(r2, __fadd_rn(r2, p0));
            r = __fmaf_rn(w, w, r);
            t[z * fs] = __fmul_rn(S[z], w);
        }
    } else {
        mid_direct(t, fs, fwd, n, false, X);
        for (int z = 0; z < n; ++z) {
            const bool k = fabsf(X[z]) > (z ? p1 : p0);
            r += k ? 1.0f : 0.0f;
            t[z * fs] = k ? X[z] : 0.0f;
        }
    }
    mid_direct(t, fs, inv, n, true, X);
    for (int z = 0; z < n; ++z) t[z * fs] = X[z];
    return r;
}

template <class T>
__device__ __forceinline__ float mid_z_any(T *v, int stride, float p0, float p1, int n, const CFArgs &a)
{
    switch (n) {
    case 1: return mid_z<1>(v, stride, p0, p1);
    case 2: return mid_z<2>(v, stride, p0, p1);
    case 4: return mid_z<4>(v, stride, p0, p1);
    case 8: return mid_z<8>(v, stride, p0, p1);
    case 16: return mid_z<16>(v, stride, p0, p1);
    case 32: return mid_z<32>(v, stride, p0, p1);
    }
    return mid_z_direct(v, stride, p0, p1, n, dtab_for(a, n, false), dtab_for(a, n, true));
}

// shared-memory floats: two tables, then the cells ([z][y][x], rows of an odd number of cells, so that
// lanes on consecutive rows fall in distinct banks)
__host__ __device__ inline int mid_smem_bytes(int BM, int B, int G, bool wiener)
{
    return 4 * (2 * BM * 16 + 8) + (wiener ? 8 : 4) * G * B * (B | 1);
}

template <int BM, bool DIRECT, bool WIENER>
__global__ void __launch_bounds__(kMidThreads, 4) cf_mid_kernel(CFArgs a)
{
    using T = std::conditional_t<WIENER, f2, float>;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int B = DIRECT ? a.B : BM, RP = B | 1, PP = B * RP, area = B * B;
    float *ft = smem, *it = smem + BM * 16, *red = it + BM * 16;
    T *cell = reinterpret_cast<T *>(red + 8);
    float *low = reinterpret_cast<float *>(cell);            // the cells' (low) words
    constexpr int W = WIENER ? 2 : 1;
    if (DIRECT) {
        const float *f = dtab_for(a, B, false), *i = dtab_for(a, B, true);
        for (int e = tid; e < BM * B; e += kMidThreads) {
            const int j = e / BM, k = e - j * BM;
            ft[e] = k < B ? f[k * B + j] : 0.0f;
            it[e] = k < B ? i[k * B + j] : 0.0f;
        }
    }
    const float rB = 1.0f / (float)B;
    auto div_b = [=](int e) { return (int)(((float)e + 0.5f) * rB); };     // e / B for small e

    for (long long grp = blockIdx.x; grp < a.ngroups; grp += gridDim.x) {
        const int n = min(a.count[grp], a.G);
        const uint32_t *pl = a.pos + grp * a.G;
        for (int p = 0; p < 3; ++p) {
            if (!a.process[p]) continue;
            __syncthreads();
            for (int k = warp; k < n; k += kMidThreads / 32) {
                const GroupLoc L = locate(a, p, grp, pl[k]);
                const float *s = L.src + (long long)L.y * a.ld + L.x, *r = L.ref + (long long)L.y * a.ld + L.x;
                for (int e = lane; e < area; e += 32) {
                    const int y = div_b(e), x = e - y * B;
                    if constexpr (WIENER) cell[k * PP + y * RP + x] = pk(__ldg(r + (long long)y * a.ld + x), __ldg(s + (long long)y * a.ld + x));
                    else cell[k * PP + y * RP + x] = __ldg(s + (long long)y * a.ld + x);
                }
            }
            __syncthreads();
            for (int t = tid; t < n * B; t += kMidThreads) mid_transform<BM, DIRECT, false>(cell + t * RP, 1, B, ft);
            __syncthreads();
            for (int t = tid; t < n * B; t += kMidThreads) {
                const int k = div_b(t), x = t - k * B;
                mid_transform<BM, DIRECT, false>(cell + k * PP + x, RP, B, ft);
            }
            __syncthreads();
            float r = 0.0f;
            for (int t = tid; t < area; t += kMidThreads) {
                const int y = div_b(t), x = t - y * B, fxy = (x == 0) + (y == 0);
                r = __fadd_rn(r, mid_z_any(cell + y * RP + x, PP, WIENER ? a.wsig2[p][n - 1] : a.thr4[p][n - 1][fxy + 1],
                                           WIENER ? 0.0f : a.thr4[p][n - 1][fxy], n, a));
            }
            r = warp_sum(r);                    // counts stay exact: at most 2^13
            if (lane == 0) red[warp] = r;
            __syncthreads();
            r = __fadd_rn(__fadd_rn(red[0], red[1]), __fadd_rn(red[2], red[3]));
            const float eps = 1.1920928955078125e-07f;
            const float denW = WIENER ? __fdiv_rn(1.0f, r > eps ? r : eps) : r < 1.0f ? 1.0f : __fdiv_rn(1.0f, r);
            if (!WIENER && a.retained && tid == 0) a.retained[(long long)p * a.ngroups + grp] = (int)r;
            const float numW = __fdiv_rn(denW, a.amp[n - 1]);
            for (int t = tid; t < n * B; t += kMidThreads) {
                const int k = div_b(t), x = t - k * B;
                mid_transform<BM, DIRECT, true>(low + W * (k * PP + x), W * RP, B, it);
            }
            __syncthreads();
            for (int t = tid; t < n * B; t += kMidThreads) mid_transform<BM, DIRECT, true>(low + W * t * RP, W, B, it);
            __syncthreads();
            for (int k = warp; k < n; k += kMidThreads / 32) {
                const GroupLoc L = locate(a, p, grp, pl[k]);
                float *d = L.num + (long long)L.y * a.ld + L.x;
                for (int e = lane; e < area; e += 32) {
                    const int y = div_b(e), x = e - y * B;
                    atomicAdd(d + (long long)y * a.ld + x, __fmul_rn(low[W * (k * PP + y * RP + x)], numW));
                }
                if (lane == 0) atomicAdd(L.wmap + (long long)L.y * a.ld + L.x, denW);
            }
        }
    }
}

}  // namespace bm3d
