// convert.cuh -- K5: per-pixel kernels around the hot path.
//   * ingest / egress: integer<->float range conversion and RGB<->OPP matrix conversion, with
//     the gains and offsets computed on the host exactly as include/Conversion.hpp:36-417 does
//     (RangeConvert, ConvertToY, MatrixConvert_RGB2YUV / _YUV2RGB, OPP branches);
//   * finalize: den = B x B box sum of the per-origin weights, out = num / den
//     (source/BM3D_Base.cpp:348-351, 455-469);
//   * VAggregate: num = sum_f num_f, den = sum_f den_f, out = num / den over the temporal window
//     (source/VAggregate.cpp:93-160, slot selection :194-202).
#pragma once

#include "common.cuh"
#include "args.h"

namespace bm3d {



__device__ __forceinline__ float clip_ref(float v, float lo, float hi)
{
    // Clip() of include/Helper.h:395-399
    return v <= lo ? lo : v >= hi ? hi : v;
}



// Eight samples of a row.  VEC: consecutive ones, read and written with 16-byte accesses where the eight fit
// in the row (8 bytes for 8-bit samples; the host checks the alignment of every plane); else
// samples t, t + rw, t + 2 rw ... of the row's rw threads, so that a warp's accesses stay contiguous.
struct RowSpan {
    int t, rw, W;
    template <bool VEC> __device__ __forceinline__ int at(int k) const { return VEC ? 8 * t + k : t + k * rw; }
};

template <bool VEC>
__device__ __forceinline__ void load8(const PlanePtr &p, int kind, int y, const RowSpan &r, float (&v)[8])
{
    const char *row = static_cast<const char *>(p.ptr) + (long long)y * p.stride;
    if (VEC && 8 * r.t + 8 <= r.W) {
        if (kind == SK_U8) {
            const uint2 q = reinterpret_cast<const uint2 *>(row)[r.t];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = (float)(((k < 4 ? q.x : q.y) >> (8 * (k & 3))) & 0xffu);
        } else if (kind == SK_U16) {
            const uint4 q = reinterpret_cast<const uint4 *>(row)[r.t];
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = (float)((w[k >> 1] >> (16 * (k & 1))) & 0xffffu);
        } else {
            const float4 a = reinterpret_cast<const float4 *>(row)[2 * r.t], b = reinterpret_cast<const float4 *>(row)[2 * r.t + 1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = r.at<VEC>(k);
        if (x >= r.W) continue;
        v[k] = kind == SK_U8 ? (float)reinterpret_cast<const uint8_t *>(row)[x]
             : kind == SK_U16 ? (float)reinterpret_cast<const uint16_t *>(row)[x] : reinterpret_cast<const float *>(row)[x];
    }
}

// integer samples by truncation, as static_cast
template <bool VEC>
__device__ __forceinline__ void store8(const PlanePtr &p, int kind, int y, const RowSpan &r, const float (&v)[8])
{
    char *row = static_cast<char *>(p.ptr) + (long long)y * p.stride;
    if (VEC && 8 * r.t + 8 <= r.W) {
        if (kind == SK_U8) {
            uint32_t w[2] = {0u, 0u};
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k >> 2] |= (uint32_t)(uint8_t)v[k] << (8 * (k & 3));
            reinterpret_cast<uint2 *>(row)[r.t] = make_uint2(w[0], w[1]);
        } else if (kind == SK_U16) {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k >> 1] |= (uint32_t)(uint16_t)v[k] << (16 * (k & 1));
            reinterpret_cast<uint4 *>(row)[r.t] = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
            reinterpret_cast<float4 *>(row)[2 * r.t] = make_float4(v[0], v[1], v[2], v[3]);
            reinterpret_cast<float4 *>(row)[2 * r.t + 1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = r.at<VEC>(k);
        if (x >= r.W) continue;
        if (kind == SK_U8) reinterpret_cast<uint8_t *>(row)[x] = (uint8_t)v[k];
        else if (kind == SK_U16) reinterpret_cast<uint16_t *>(row)[x] = (uint16_t)v[k];
        else reinterpret_cast<float *>(row)[x] = v[k];
    }
}

__device__ __forceinline__ float linear_ref(float t, const LinearOp &o)
{
    t = __fadd_rn(__fmul_rn(t, o.gain), o.offset);
    return o.clip ? clip_ref(t, o.lo, o.hi) : t;
}

// One thread per eight samples of a row, one grid row per frame; the planes' addresses come with the launch.
// Bound: HBM.  4 frames of 1920x1080 RGB, 16 bits -> float OPP -> 16 bits, 300 MB with the intermediate: a pixel per
// thread and address tables copied to the device first 97 us, 54 us now.
template <bool VEC>
__global__ void __launch_bounds__(256) convert_kernel(const __grid_constant__ ConvProgram pr, const __grid_constant__ ConvTable tab)
{
    const int rw = (pr.W + 7) >> 3, u = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = u / rw, f = blockIdx.y;
    if (y >= pr.H) return;
    const RowSpan r{u - y * rw, rw, pr.W};
    const int i0 = f * pr.nin, o0 = f * pr.nout;
    if (pr.raw || pr.mode == 0) {
        for (int c = 0; c < pr.nin; ++c) {
            if (!tab.out[o0 + c].ptr) continue;
            float v[8];
            load8<VEC>(tab.in[i0 + c], pr.in_kind, y, r, v);
            if (!pr.raw) {
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = linear_ref(v[k], pr.op[c]);
            }
            store8<VEC>(tab.out[o0 + c], pr.out_kind, y, r, v);
        }
        return;
    }
    float a[8], b[8], c[8];
    load8<VEC>(tab.in[i0], pr.in_kind, y, r, a);
    load8<VEC>(tab.in[i0 + 1], pr.in_kind, y, r, b);
    load8<VEC>(tab.in[i0 + 2], pr.in_kind, y, r, c);
    if (pr.mode == 1 || pr.mode == 2) {
        float Y[8], U[8], V[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            Y[k] = linear_ref(__fadd_rn(__fadd_rn(a[k], b[k]), c[k]), pr.op[0]);
            U[k] = linear_ref(__fsub_rn(a[k], c[k]), pr.op[1]);
            V[k] = linear_ref(__fadd_rn(__fsub_rn(a[k], __fmul_rn(b[k], 2.0f)), c[k]), pr.op[2]);
        }
        store8<VEC>(tab.out[o0], pr.out_kind, y, r, Y);
        if (pr.mode == 1) {
            if (tab.out[o0 + 1].ptr) store8<VEC>(tab.out[o0 + 1], pr.out_kind, y, r, U);
            if (tab.out[o0 + 2].ptr) store8<VEC>(tab.out[o0 + 2], pr.out_kind, y, r, V);
        }
        return;
    }
    const float *m = pr.coef;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float Y = a[k], U = b[k], V = c[k];
        a[k] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], Y), __fmul_rn(m[1], U)), __fmul_rn(m[2], V)), pr.off[0]);
        b[k] = __fadd_rn(__fadd_rn(__fmul_rn(m[3], Y), __fmul_rn(m[5], V)), pr.off[1]);
        c[k] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[6], Y), __fmul_rn(m[7], U)), __fmul_rn(m[8], V)), pr.off[2]);
        if (pr.op[0].clip) {
            a[k] = clip_ref(a[k], pr.op[0].lo, pr.op[0].hi);
            b[k] = clip_ref(b[k], pr.op[0].lo, pr.op[0].hi);
            c[k] = clip_ref(c[k], pr.op[0].lo, pr.op[0].hi);
        }
    }
    store8<VEC>(tab.out[o0], pr.out_kind, y, r, a);
    store8<VEC>(tab.out[o0 + 1], pr.out_kind, y, r, b);
    store8<VEC>(tab.out[o0 + 2], pr.out_kind, y, r, c);
}

// Tile of the denominator (the B x B box sum of the per-origin weight map wm) for output rows
// [ty0, ty0 + kFinTH) and columns [tx0, tx0 + kFinTW): the weight region with its (B - 1) halo is
// staged in shared memory, summed along x, then along y (2B additions per pixel instead of B^2).
// On return den[r * kFinTW + c] holds the denominator of pixel (ty0 + r, tx0 + c).
constexpr int kFinTH = 32, kFinTW = 64;

__host__ __device__ inline int finalize_smem_floats(int B)
{
    if (B == 8) return (kFinTH + 7) * (kFinTW + 8) + (kFinTH + 7) * kFinTW;
    return (kFinTH + B - 1) * (kFinTW + B - 1) + (kFinTH + B - 1) * kFinTW + kFinTH * kFinTW;
}

__device__ __forceinline__ float *box_den_tile(float *sm, const float *wm, int ld, int H, int W, int B, int ty0, int tx0)
{
    const int RH = kFinTH + B - 1, RW = kFinTW + B - 1;
    float *reg = sm;
    float *hs = sm + RH * RW;
    float *den = hs + RH * kFinTW;
    for (int e = threadIdx.x; e < RH * RW; e += blockDim.x) {
        const int r = e / RW, c = e - r * RW;
        const int yy = ty0 - (B - 1) + r, xx = tx0 - (B - 1) + c;
        reg[e] = (yy >= 0 && xx >= 0 && yy < H && xx < W) ? wm[(long long)yy * ld + xx] : 0.0f;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < RH * kFinTW; e += blockDim.x) {
        const int r = e / kFinTW, c = e - r * kFinTW;
        float v = 0.0f;
        for (int k = 0; k < B; ++k) v = __fadd_rn(v, reg[r * RW + c + k]);
        hs[e] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kFinTH * kFinTW; e += blockDim.x) {
        const int r = e / kFinTW, c = e - r * kFinTW;
        float v = 0.0f;
        for (int k = 0; k < B; ++k) v = __fadd_rn(v, hs[(r + k) * kFinTW + c]);
        den[e] = v;
    }
    __syncthreads();
    return den;
}

// The same for B = 8, without the tile of denominators: the weight region is staged in 16-byte chunks from
// column tx0 - 8 on, a thread sums four neighbouring columns along x, then its column's eight rows along y out
// of fifteen row sums, and hands use(row, denominator).  Additions in the same order.
// Bound: HBM.  24 planes of 1920x1080: 405 us with the generic form (a division per element of every stage,
// four passes over shared memory), 178 us here.
constexpr int kFin8Pitch = kFinTW + 8;

template <class Use>
__device__ __forceinline__ void box_den_8(float *reg, float *hs, const float *wm, int ld, int H, int ty0, int tx0, Use &&use)
{
    constexpr int RH = kFinTH + 7, Q = kFin8Pitch / 4;
    for (int e = threadIdx.x; e < RH * Q; e += 256) {
        const int r = e / Q, c = 4 * (e - r * Q);
        const int yy = ty0 - 7 + r, xx = tx0 - 8 + c;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (yy >= 0 && yy < H && xx >= 0 && xx < ld) v = *reinterpret_cast<const float4 *>(wm + (long long)yy * ld + xx);
        *reinterpret_cast<float4 *>(reg + r * kFin8Pitch + c) = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < RH * (kFinTW / 4); e += 256) {
        const int r = e / (kFinTW / 4), c = 4 * (e % (kFinTW / 4));
        float w[12];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float4 v = *reinterpret_cast<const float4 *>(reg + r * kFin8Pitch + c + 4 * k);
            w[4 * k] = v.x;
            w[4 * k + 1] = v.y;
            w[4 * k + 2] = v.z;
            w[4 * k + 3] = v.w;
        }
        float o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o[i] = 0.0f;
#pragma unroll
            for (int k = 1; k <= 8; ++k) o[i] = __fadd_rn(o[i], w[i + k]);
        }
        *reinterpret_cast<float4 *>(hs + r * kFinTW + c) = make_float4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
    const int c = threadIdx.x & (kFinTW - 1), r0 = 8 * (threadIdx.x / kFinTW);
    float h[15];
#pragma unroll
    for (int k = 0; k < 15; ++k) h[k] = hs[(r0 + k) * kFinTW + c];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float v = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v = __fadd_rn(v, h[i + k]);
        use(i, ty0 + r0 + i, tx0 + c, v);
    }
}

// grid (tiles along x, tiles along y, frames * 3 planes)
__global__ void __launch_bounds__(256) finalize_kernel(const __grid_constant__ FinalizeArgs a)
{
    extern __shared__ __align__(16) float fsm[];
    const int f = blockIdx.z / 3, p = blockIdx.z % 3;
    if (!a.process[p]) return;
    const int ty0 = blockIdx.y * kFinTH, tx0 = blockIdx.x * kFinTW;
    const long long fo = (long long)f * a.frame_stride;
    if (a.B == 8) {
        // the thread's numerators are on their way during the sums
        const float *nm = a.num[p] + fo;
        float *o = a.out[p] + fo;
        const int x = tx0 + (int)(threadIdx.x & (kFinTW - 1)), yb = ty0 + 8 * (int)(threadIdx.x / kFinTW);
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (yb + i < a.H && x < a.W) v[i] = nm[(long long)(yb + i) * a.ld + x];
        box_den_8(fsm, fsm + (kFinTH + 7) * kFin8Pitch, a.wmap[p] + fo, a.ld, a.H, ty0, tx0, [&](int i, int y, int xx, float den) {
            if (y < a.H && xx < a.W) o[(long long)y * a.ld + xx] = __fdiv_rn(v[i], den);
        });
        return;
    }
    const float *den = box_den_tile(fsm, a.wmap[p] + fo, a.ld, a.H, a.W, a.B, ty0, tx0);
    const float *nm = a.num[p] + fo;
    float *o = a.out[p] + fo;
    for (int e = threadIdx.x; e < kFinTH * kFinTW; e += blockDim.x) {
        const int r = e / kFinTW, c = e - r * kFinTW;
        const int y = ty0 + r, x = tx0 + c;
        if (y < a.H && x < a.W) o[(long long)y * a.ld + x] = __fdiv_rn(nm[(long long)y * a.ld + x], den[e]);
    }
}


__global__ void vaggregate_kernel(VAggArgs a)
{
    const int f = blockIdx.z;
    const int p = blockIdx.y % 3;
    if (!a.process[p]) return;
    const int y = blockIdx.y / 3;
    const int frames = a.nframes[f];
    const int boff = a.b_off[f];
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < a.W; x += gridDim.x * blockDim.x) {
        float num = 0.0f, den = 0.0f;
        for (int i = 0, o = a.radius - boff; i < frames; ++i, --o) {
            const PlanePtr &pp = a.in[(f * a.frames_max + i) * 3 + p];
            const char *base = static_cast<const char *>(pp.ptr);
            const float *nrow = reinterpret_cast<const float *>(base + ((long long)o * 2 * a.H + y) * pp.stride);
            const float *drow = reinterpret_cast<const float *>(base + ((long long)(o * 2 + 1) * a.H + y) * pp.stride);
            num = __fadd_rn(num, nrow[x]);
            den = __fadd_rn(den, drow[x]);
        }
        a.out[p][(long long)f * a.frame_stride + (long long)y * a.ld + x] = __fdiv_rn(num, den);
    }
}

// grid (tiles along x, slots * tiles along y, frames * 3 planes)
__global__ void __launch_bounds__(256) vstack_kernel(const __grid_constant__ VStackArgs a)
{
    extern __shared__ __align__(16) float fsm[];
    const int f = blockIdx.z / 3;
    const int p = blockIdx.z % 3;
    if (!a.process[p]) return;
    const int tiles_y = (a.H + kFinTH - 1) / kFinTH;
    const int s = blockIdx.y / tiles_y;
    const int ty0 = (blockIdx.y - s * tiles_y) * kFinTH, tx0 = blockIdx.x * kFinTW;
    const long long so = ((long long)f * a.slots + s) * a.slot_stride;
    if (a.B == 8) {
        const float *nm = a.num[p] + so;
        const PlanePtr &o = a.out[f * 3 + p];
        float *nrow = reinterpret_cast<float *>(static_cast<char *>(o.ptr) + (long long)(2 * s) * a.H * o.stride);
        float *drow = reinterpret_cast<float *>(static_cast<char *>(o.ptr) + (long long)(2 * s + 1) * a.H * o.stride);
        const long long stride = o.stride >> 2;
        const int x = tx0 + (int)(threadIdx.x & (kFinTW - 1)), yb = ty0 + 8 * (int)(threadIdx.x / kFinTW);
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (yb + i < a.H && x < a.W) v[i] = nm[(long long)(yb + i) * a.ld + x];
        box_den_8(fsm, fsm + (kFinTH + 7) * kFin8Pitch, a.wmap[p] + so, a.ld, a.H, ty0, tx0, [&](int i, int y, int xx, float den) {
            if (y >= a.H || xx >= a.W) return;
            nrow[(long long)y * stride + xx] = v[i];
            drow[(long long)y * stride + xx] = den;
        });
        return;
    }
    const float *den = box_den_tile(fsm, a.wmap[p] + so, a.ld, a.H, a.W, a.B, ty0, tx0);
    const float *nm = a.num[p] + so;
    const PlanePtr &o = a.out[f * 3 + p];
    for (int e = threadIdx.x; e < kFinTH * kFinTW; e += blockDim.x) {
        const int r = e / kFinTW, c = e - r * kFinTW;
        const int y = ty0 + r, x = tx0 + c;
        if (y >= a.H || x >= a.W) continue;
        float *nrow = reinterpret_cast<float *>(static_cast<char *>(o.ptr) + ((long long)(2 * s) * a.H + y) * o.stride);
        float *drow = reinterpret_cast<float *>(static_cast<char *>(o.ptr) + ((long long)(2 * s + 1) * a.H + y) * o.stride);
        nrow[x] = nm[(long long)y * a.ld + x];
        drow[x] = den[e];
    }
}

}  // namespace bm3d
