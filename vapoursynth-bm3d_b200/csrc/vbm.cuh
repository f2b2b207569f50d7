// vbm.cuh -- K2: V-BM3D spatio-temporal grouping (predictive search).
//
// Replaces VBM3D_Process_Base::BlockMatching (source/VBM3D_Base.cpp:540-659):
//   1. full search in the current frame (K1 semantics, reference pinned first);
//   2. the first ps_num entries of that list (reference included) seed the predictive search:
//      GenSearchPos builds the sorted, de-duplicated union of (2*ps_range/ps_step+1)^2 windows
//      around them (include/Block.h:771-827);
//   3. frames cur-1 .. 0 and then cur+1 .. last are searched over such unions, each frame seeded
//      by the previous frame's best ps_num (the first step of each direction uses the current
//      frame's union); per frame the matches with 0 < dist <= thSSE are kept, partial_sort-ed to
//      group_size when more survive, stable_sort-ed otherwise (include/Block.h:655-677);
//   4. the concatenation [current, backward..., forward...] is partial_sort-ed from the second
//      entry when longer than group_size (source/VBM3D_Base.cpp:652-656).
// One warp per reference block.  The current-frame list comes from K1 (run with keys); this
// kernel performs steps 2-4.
#pragma once

#include "select.cuh"
#include "args.h"
#include "bm.cuh"
#include "proposal.cuh"

namespace bm3d {


__device__ __forceinline__ float ssd8_global(const float (&rb)[64], const float *src, int ld)
{
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int y = 0; y < 8; ++y) {
        const float *g = src + (long long)y * ld;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float d = __fsub_rn(rb[y * 8 + k], __ldg(g + k));
            acc[k] = __fadd_rn(acc[k], __fmul_rn(d, d));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float d = __fsub_rn(rb[y * 8 + 4 + k], __ldg(g + 4 + k));
            acc[k] = __fadd_rn(acc[k], __fmul_rn(d, d));
        }
    }
    return lane_combine(acc);
}

__device__ __forceinline__ float ssd_any_global(const float *rblk, int B, const float *src, int ld)
{
    const int res = B % 8, simdw = B - res;
    float dist = 0.0f;
    if (simdw > 0) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int y = 0; y < B; ++y)
            for (int c0 = 0; c0 < simdw; c0 += 8) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = __fsub_rn(rblk[y * B + c0 + k], __ldg(src + (long long)y * ld + c0 + k));
                    acc[k] = __fadd_rn(acc[k], __fmul_rn(d, d));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float d = __fsub_rn(rblk[y * B + c0 + 4 + k], __ldg(src + (long long)y * ld + c0 + 4 + k));
                    acc[k] = __fadd_rn(acc[k], __fmul_rn(d, d));
                }
            }
        dist = __fadd_rn(dist, lane_combine(acc));
    }
    for (int y = 0; y < B; ++y)
        for (int x = simdw; x < B; ++x) {
            const float d = __fsub_rn(rblk[y * B + x], __ldg(src + (long long)y * ld + x));
            dist = __fadd_rn(dist, __fmul_rn(d, d));
        }
    return dist;
}

// Union of lattice windows around `nc` centres, sorted by (y, x) and de-duplicated, written
// to sp (packed y<<16|x).  Returns the count.  Warp-cooperative: the union is built as a
// sorted merge, one centre at a time, mirroring MergeSearchPos + unique.
__device__ int gen_search_pos_warp(const uint32_t *centres, int nc, int H, int W, int B, int range,
                                   int step, uint32_t *sp, uint32_t *tmp, int cap)
{
    const int lane = (int)lane_id();
    int n = 0;
    for (int ci = 0; ci < nc; ++ci) {
        const int cy = unpack_y(centres[ci]), cx = unpack_x(centres[ci]);
        const int l = search_boundary(cx, 0, range, step);
        const int r = search_boundary(cx, W - B, range, step);
        const int t = search_boundary(cy, 0, range, step);
        const int b = search_boundary(cy, H - B, range, step);
        const int ncol = (r - l) / step + 1;
        const int nrow = (b - t) / step + 1;
        const int nw = ncol * nrow;
        // merge sp[0..n) with the window (both sorted) into tmp, keeping duplicates out
        // rank of each element in the other list gives its merged position
        int total = 0;
        for (int k = lane; k < n; k += 32) {
            const uint32_t v = sp[k];
            // count window elements < v
            const int vy = unpack_y(v), vx = unpack_x(v);
            int rows_before = vy <= t ? 0 : vy > b ? nrow : (vy - t + step - 1) / step;
            int cnt = rows_before * ncol;
            if (vy >= t && vy <= b && (vy - t) % step == 0) {
                int cols_before = vx <= l ? 0 : vx > r ? ncol : (vx - l + step - 1) / step;
                cnt += cols_before;
            }
            tmp[k + cnt] = v;
        }
        for (int k = lane; k < nw; k += 32) {
            const int ry = k / ncol, cc = k - ry * ncol;
            const uint32_t v = pack_yx(t + ry * step, l + cc * step);
            // count sp elements <= v (equal elements from the first range come first)
            int lo = 0, hi = n;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (sp[mid] <= v) lo = mid + 1; else hi = mid;
            }
            tmp[k + lo] = v;
        }
        total = n + nw;
        __syncwarp();
        // unique (adjacent duplicates) while copying back
        int out = 0;
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + lane;
            bool keep = false;
            uint32_t v = 0;
            if (k < total) {
                v = tmp[k];
                keep = k == 0 || tmp[k - 1] != v;
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int d = out + __popc(m & ((1u << lane) - 1u));
                if (d < cap) sp[d] = v;
            }
            out += __popc(m);
        }
        __syncwarp();
        n = out < cap ? out : cap;
    }
    return n;
}

// Per-frame selection of the search-position form: partial_sort(begin, begin + G) when more
// than G survive, stable_sort otherwise.  Keys computed for all valid (invalid = -1).
// Result (sorted keys + scan indices) in hk/hi; returns the count.
__device__ int select_positions(float *sk, int ns, int G, float *hk, int *hi)
{
    const int lane = (int)lane_id();
    int cnt = 0;
    for (int c = lane; c < ns; c += 32) cnt += sk[c] >= 0.0f;
    const int nvalid = warp_sum(cnt);
    int n = 0;
    if (lane == 0) {
        if (nvalid > G) {
            int c = 0;
            for (; c < ns && n < G; ++c)
                if (sk[c] >= 0.0f) { hk[n] = sk[c]; hi[n] = c; ++n; }
            heap_make(hk, hi, G);
            for (; c < ns; ++c)
                if (sk[c] >= 0.0f) heap_offer(hk, hi, G, sk[c], c);
            heap_sort(hk, hi, G);
        } else {
            for (int c = 0; c < ns; ++c)
                if (sk[c] >= 0.0f) { hk[n] = sk[c]; hi[n] = c; ++n; }
            stable_sort_keys(hk, hi, n);
        }
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    __syncwarp();
    return n;
}

__global__ void __launch_bounds__(128) vbm_predict_kernel(VBMArgs a)
{
    extern __shared__ float smem[];
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5;
    const int f = blockIdx.z;
    const int by = blockIdx.y;
    const int bx = blockIdx.x * a.warps + warp;
    if (bx >= a.nbx) return;

    // per-warp shared layout
    const int per_warp = vbm_warp_floats(a.sp_cap, a.list_cap, a.G, a.ps_num, a.B);
    float *base = smem + (size_t)warp * per_warp;
    uint32_t *sp = reinterpret_cast<uint32_t *>(base);
    uint32_t *tmp = sp + a.sp_cap;
    float *sk = reinterpret_cast<float *>(tmp + vbm_tmp_cap(a.sp_cap));
    float *lk = sk + a.sp_cap;                                  // concatenated keys
    uint32_t *lp = reinterpret_cast<uint32_t *>(lk + a.list_cap); // concatenated positions (zyx)
    float *fk = reinterpret_cast<float *>(lp + a.list_cap);     // per-frame selection keys
    int *fi = reinterpret_cast<int *>(fk + a.list_cap);
    uint32_t *cen = reinterpret_cast<uint32_t *>(fi + a.list_cap);
    float *hk = reinterpret_cast<float *>(cen + a.ps_num);
    int *hi = reinterpret_cast<int *>(hk + a.G);
    float *rblk = reinterpret_cast<float *>(hi + a.G);

    const int frames = a.win_len[f];
    const int cur = a.win_cur[f];
    const int wbase = a.win_base[f];
    const int B = a.B;
    const int G = a.G;
    const int j = a.scan_y[by], i = a.scan_x[bx];
    const size_t ob = ((size_t)f * a.nby + by) * a.nbx + bx;
    const float *curplane = a.ref + (long long)(wbase + cur) * a.frame_stride;

    // current-frame list
    const int n0 = a.cur_n[ob];
    int L = 0;
    for (int k = lane; k < n0; k += 32) {
        const uint32_t p = a.cur_pos[ob * G + k];
        lp[k] = pack_zyx(cur, unpack_y(p), unpack_x(p));
        lk[k] = a.cur_key[ob * G + k];
    }
    L = n0;
    if (G == 1) {
        if (lane == 0) {
            a.out_pos[ob * G] = pack_zyx(cur, j, i);
            if (a.out_key) a.out_key[ob * G] = 0.0f;
            a.out_n[ob] = 1;
        }
        return;
    }
    for (int idx = lane; idx < B * B; idx += 32) {
        const int y = idx / B, x = idx - y * B;
        rblk[idx] = curplane[(long long)(j + y) * a.ld + i + x];
    }
    __syncwarp();
    float rb[64];
    if (B == 8) {
#pragma unroll
        for (int e = 0; e < 64; ++e) rb[e] = rblk[e];
    }

    // learned proposals: descriptor of the reference block (current frame)
    const __nv_bfloat16 *dsc = static_cast<const __nv_bfloat16 *>(a.desc);
    const int Wd = a.W - 7;
    float da[kPropCh];
    if (dsc) load_desc(dsc + (long long)(wbase + cur) * a.desc_frame * kPropCh, (long long)j * Wd + i, da);

    // seeds from the current frame
    const int ncen0 = min(a.ps_num, n0);
    for (int k = lane; k < ncen0; k += 32) {
        const uint32_t p = a.cur_pos[ob * G + k];
        cen[k] = p;
    }
    __syncwarp();

    for (int dir = -1; dir <= 1; dir += 2) {
        int ncen = ncen0;
        if (dir == 1) {
            for (int k = lane; k < ncen0; k += 32) cen[k] = a.cur_pos[ob * G + k];
            __syncwarp();
        }
        for (int fz = cur + dir; fz >= 0 && fz < frames; fz += dir) {
            const int ns = gen_search_pos_warp(cen, ncen, a.H, a.W, B, a.ps_range, a.ps_step, sp, tmp, a.sp_cap);
            const float *plane = a.ref + (long long)(wbase + fz) * a.frame_stride;
            if (dsc && B == 8 && ns > a.nprop) {
                // learned proposals: the nprop positions of smallest descriptor distance (ties by
                // position order) get exact distances, the others are left out of this frame's list
                const __nv_bfloat16 *dz = dsc + (long long)(wbase + fz) * a.desc_frame * kPropCh;
                for (int c = lane; c < ns; c += 32) {
                    float dc[kPropCh];
                    load_desc(dz, (long long)unpack_y(sp[c]) * Wd + unpack_x(sp[c]), dc);
                    float sc = 0.0f;
#pragma unroll
                    for (int k = 0; k < kPropCh; ++k) sc = fmaf(da[k] - dc[k], da[k] - dc[k], sc);
                    sk[c] = sc;
                }
                __syncwarp();
                // the nprop smallest (score, position index) by radix selection (tmp is free here)
                int rank = a.nprop - 1;
                const uint32_t cutv = warp_radix_cut(sk, ns, rank, reinterpret_cast<int *>(tmp));
                const unsigned lt = (1u << lane) - 1u;
                int eq = 0;
                for (int c0 = 0; c0 < ns; c0 += 32) {
                    const int c = c0 + lane;
                    const uint32_t u = c < ns ? __float_as_uint(sk[c]) : 0xffffffffu;
                    const bool isq = c < ns && u == cutv;
                    const unsigned mq = __ballot_sync(0xffffffffu, isq);
                    const bool in = c < ns && (u < cutv || (isq && eq + __popc(mq & lt) <= rank));
                    eq += __popc(mq);
                    if (c < ns) {
                        float key = -1.0f;
                        if (in) {
                            const float d = ssd8_global(rb, plane + (long long)unpack_y(sp[c]) * a.ld + unpack_x(sp[c]), a.ld);
                            key = dist_valid(d, a.thSSE) ? dist_to_key(d, a.distMul) : -1.0f;
                        }
                        sk[c] = key;
                    }
                }
            } else {
                for (int c = lane; c < ns; c += 32) {
                    const int y = unpack_y(sp[c]), x = unpack_x(sp[c]);
                    const float *src = plane + (long long)y * a.ld + x;
                    const float d = B == 8 ? ssd8_global(rb, src, a.ld) : ssd_any_global(rblk, B, src, a.ld);
                    sk[c] = dist_valid(d, a.thSSE) ? dist_to_key(d, a.distMul) : -1.0f;
                }
            }
            __syncwarp();
            const int nf = select_positions(sk, ns, G, fk, fi);
            for (int k = lane; k < nf; k += 32) {
                const uint32_t p = sp[fi[k]];
                if (L + k < a.list_cap) {
                    lp[L + k] = pack_zyx(fz, unpack_y(p), unpack_x(p));
                    lk[L + k] = fk[k];
                }
            }
            // next seeds: first ps_num of this frame's list
            const int nn = min(a.ps_num, nf);
            __syncwarp();
            for (int k = lane; k < nn; k += 32) cen[k] = sp[fi[k]];
            ncen = nn;
            L += nf;
            __syncwarp();
        }
    }
    if (L > a.list_cap) L = a.list_cap;

    // final merge: partial_sort(begin + 1, begin + G) if longer than G
    uint32_t *op = a.out_pos + ob * G;
    float *ok = a.out_key ? a.out_key + ob * G : nullptr;
    if (L > G) {
        if (lane == 0) {
            const int K = G - 1;
            for (int k = 0; k < K; ++k) { hk[k] = lk[1 + k]; hi[k] = 1 + k; }
            heap_make(hk, hi, K);
            for (int c = 1 + K; c < L; ++c) heap_offer(hk, hi, K, lk[c], c);
            heap_sort(hk, hi, K);
            op[0] = lp[0];
            if (ok) ok[0] = lk[0];
            for (int k = 0; k < K; ++k) {
                op[1 + k] = lp[hi[k]];
                if (ok) ok[1 + k] = hk[k];
            }
            a.out_n[ob] = G;
        }
    } else {
        for (int k = lane; k < L; k += 32) {
            op[k] = lp[k];
            if (ok) ok[k] = lk[k];
        }
        if (lane == 0) a.out_n[ob] = L;
    }
}

// ---- B = 8, step-1 search around at most two centres: register-blocked distances, parallel selection --
//
// The general kernel above spends nine tenths of its time outside the distances: a sorted union
// built by binary searches, and single-lane heaps over every candidate.  Here the union is split
// in closed form (centre 0's window; centre 1's rows outside it; centre 1's columns outside it in
// the shared rows), a lane computes four adjacent candidates at a time from a window staged in
// shared memory, and the best G are taken by warp minimum reductions.  The scan order of the
// union only decides between equal keys: a search whose kept keys, or the key at the cut, are not
// distinct is redone by the general routines.
// Bound: FP32 issue of the distances.  1280x720 x 7 frames, radius 3, 169 to 338 candidates per
// search: predictive search 77.9 ms before, 13.5 ms now; 1920x1080 x 5 frames, radius 1,
// 81 to 162 candidates: 4.74 -> 1.02 ms.  (With windows by rows, whose packed pairs of columns have to be
// re-packed by moves for every other candidate: 15.0 and 1.10 ms.)

// Exact distances and the reference's selection over one frame's union: keys and positions of the
// frame's list into fk / fp; returns its length.
__device__ __noinline__ int vbm_frame_general(const VBMArgs &a, const float *rblk, const float *plane, const uint32_t *cen,
                                              int ncen, float *work, float *fk, uint32_t *fp)
{
    const int lane = (int)lane_id();
    uint32_t *sp = reinterpret_cast<uint32_t *>(work);
    uint32_t *tmp = sp + vbm_tmp_cap(a.sp_cap);
    float *sk = reinterpret_cast<float *>(tmp + vbm_tmp_cap(a.sp_cap));
    __syncwarp();
    const int ns = gen_search_pos_warp(cen, ncen, a.H, a.W, 8, a.ps_range, a.ps_step, sp, tmp, a.sp_cap);
    for (int c = lane; c < ns; c += 32) {
        const float d = ssd_any_global(rblk, 8, plane + (long long)unpack_y(sp[c]) * a.ld + unpack_x(sp[c]), a.ld);
        sk[c] = dist_valid(d, a.thSSE) ? dist_to_key(d, a.distMul) : -1.0f;
    }
    __syncwarp();
    int *fi = reinterpret_cast<int *>(fp);
    const int nf = select_positions(sk, ns, a.G, fk, fi);
    for (int k = lane; k < nf; k += 32) fp[k] = sp[fi[k]];
    __syncwarp();
    return nf;
}

// A lane's two smallest values and their slots, out of a lane-private column
struct LaneBest {
    float b1, b2;
    int s1, s2;
    __device__ __forceinline__ void clear() { b1 = b2 = __int_as_float(0x7f800000); s1 = s2 = 0; }
    __device__ __forceinline__ void offer(float d, int s)
    {
        if (d < b1) { b2 = b1; s2 = s1; b1 = d; s1 = s; }
        else if (d < b2) { b2 = d; s2 = s; }
    }
};

// The G + 1 smallest values of the warp's columns (col[s * 32], s < nslots, +inf where invalid; `left`
// valid ones in the lane's own) in ascending order: rank k < G ends in lane k's `d`, `own` (the lane
// that held it) and `slot`; returns how many there are up to G, *cut = the rank-G value (+inf if none).
// Equal values keep both entries, in any order.
__device__ __forceinline__ int warp_smallest(LaneBest &lb, float *col, int nslots, int left, int G, float &d, int &own, int &slot,
                                             float &cut)
{
    const int lane = (int)lane_id();
    const unsigned inf = 0x7f800000u;
    d = cut = __uint_as_float(inf);
    own = slot = 0;
    int n = 0;
    for (int k = 0; k <= G; ++k) {
        const unsigned m = __reduce_min_sync(0xffffffffu, __float_as_uint(lb.b1));
        if (m == inf) break;
        if (k == G) {
            cut = __uint_as_float(m);
            break;
        }
        const int o = __ffs(__ballot_sync(0xffffffffu, __float_as_uint(lb.b1) == m)) - 1;
        const int so = __shfl_sync(0xffffffffu, lb.s1, o);
        if (lane == k) { d = __uint_as_float(m); own = o; slot = so; }
        ++n;
        if (lane == o) {
            col[lb.s1 * 32] = __uint_as_float(inf);
            --left;
            lb.b1 = lb.b2;
            lb.s1 = lb.s2;
            lb.b2 = __uint_as_float(inf);
            if (__float_as_uint(lb.b1) == inf && left > 0) {
                lb.clear();
                for (int s = 0; s < nslots; ++s) lb.offer(col[s * 32], s);
            }
        }
    }
    return n;
}

__global__ void __launch_bounds__(128, 5) vbm_predict8_kernel(VBMArgs a)
{
    extern __shared__ __align__(16) float smem[];
    const int lane = (int)lane_id();
    const int warp = threadIdx.x >> 5;
    const int f = blockIdx.z;
    const int by = blockIdx.y;
    const int bx = blockIdx.x * a.warps + warp;
    if (bx >= a.nbx) return;

    const int R = a.ps_range, G = a.G;
    const int P = vbm8_pitch(R);
    float *rblk = smem + (size_t)warp * vbm8_warp_floats(R, a.sp_cap, a.list_cap, G);
    f32x2 *rpair = reinterpret_cast<f32x2 *>(rblk + 64);
    float *work = rblk + 128;
    f32x2 *patch0 = reinterpret_cast<f32x2 *>(work), *patch1 = reinterpret_cast<f32x2 *>(work + vbm8_patch_floats(R));
    const int odd = vbm8_odd(R);
    float *col = work + 2 * vbm8_patch_floats(R) + lane;
    float *lk = work + vbm8_work_floats(R, a.sp_cap, a.list_cap);
    uint32_t *lp = reinterpret_cast<uint32_t *>(lk + a.list_cap);
    float *fk = reinterpret_cast<float *>(lp + a.list_cap);
    uint32_t *fp = reinterpret_cast<uint32_t *>(fk + G);
    uint32_t *cen = fp + G;

    const int frames = a.win_len[f];
    const int cur = a.win_cur[f];
    const int wbase = a.win_base[f];
    const int j = a.scan_y[by], i = a.scan_x[bx];
    const size_t ob = ((size_t)f * a.nby + by) * a.nbx + bx;
    const float *curplane = a.ref + (long long)(wbase + cur) * a.frame_stride;
    const float inf = __int_as_float(0x7f800000);

    const int n0 = a.cur_n[ob];
    int L = n0;
    for (int k = lane; k < n0; k += 32) {
        const uint32_t p = a.cur_pos[ob * G + k];
        lp[k] = pack_zyx(cur, unpack_y(p), unpack_x(p));
        lk[k] = a.cur_key[ob * G + k];
    }
    if (G == 1) {
        if (lane == 0) {
            a.out_pos[ob * G] = pack_zyx(cur, j, i);
            if (a.out_key) a.out_key[ob * G] = 0.0f;
            a.out_n[ob] = 1;
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < 64; e += 32) {
        const int idx = e + lane;
        const float v = curplane[(long long)(j + (idx >> 3)) * a.ld + i + (idx & 7)];
        rblk[idx] = v;
        reinterpret_cast<float *>(rpair + (idx >> 4) * 8 + (idx & 7))[(idx >> 3) & 1] = v;
    }
    // window rows [t, t + rows), columns l .. l + cols - 1 of a plane to a patch, twice: as pairs of rows from even
    // and from odd ones
    auto stage = [&](f32x2 *patch, const float *plane, int t, int l, int rows, int cols) {
        if (lane >= cols) return;
        const float *src = plane + (long long)t * a.ld + l + lane;
        float *e = reinterpret_cast<float *>(patch + lane), *o = reinterpret_cast<float *>(patch + odd + lane);
        // rows 2q and 2q + 1: the halves of even pair q; the second half of odd pair q - 1 and the first of pair q
        // (the last window row starts no pair)
        for (int q = 0; 2 * q < rows; ++q, src += 2 * a.ld, e += 2 * P, o += 2 * P) {
            tc::cp_async4(e, src);
            if (q > 0) tc::cp_async4(o - 2 * P + 1, src);
            if (2 * q + 1 < rows) tc::cp_async4(e + 1, src + a.ld);
            if (2 * q + 2 < rows) tc::cp_async4(o, src + a.ld);
        }
    };

    const int ncen0 = min(a.ps_num, n0);
    for (int dir = -1; dir <= 1; dir += 2) {
        int ncen = ncen0;
        uint32_t c0 = a.cur_pos[ob * G], c1 = ncen0 > 1 ? a.cur_pos[ob * G + 1] : 0u;
        for (int fz = cur + dir; fz >= 0 && fz < frames && ncen > 0; fz += dir) {
            const float *plane = a.ref + (long long)(wbase + fz) * a.frame_stride;
            // windows [t, b] x [l, r] of the centres (step 1: the clamped range)
            const int y0 = unpack_y(c0), x0 = unpack_x(c0), y1 = unpack_y(c1), x1 = unpack_x(c1);
            const int t0 = max(0, y0 - R), b0 = min(a.H - 8, y0 + R), l0 = max(0, x0 - R), r0 = min(a.W - 8, x0 + R);
            const int t1 = max(0, y1 - R), b1 = min(a.H - 8, y1 + R), l1 = max(0, x1 - R), r1 = min(a.W - 8, x1 + R);
            __syncwarp();
            stage(patch0, plane, t0, l0, b0 - t0 + 8, r0 - l0 + 8);
            // centre 1's candidates outside centre 0's window: rows [at, at + an) whole, rows
            // [it, it + in) of both windows in the columns [bl, bl + bn) only
            int at = t1, an = 0, it = 0, in = 0, bl = l1, bn = 0;
            if (ncen > 1) {
                stage(patch1, plane, t1, l1, b1 - t1 + 8, r1 - l1 + 8);
                if (t1 > b0 || b1 < t0) an = b1 - t1 + 1;
                else if (y1 >= y0) {          // the clamped windows keep the centres' order
                    it = t1; in = min(b0, b1) - t1 + 1;
                    at = b0 + 1; an = max(0, b1 - b0);
                } else {
                    it = t0; in = b1 - t0 + 1;
                    an = t0 - t1;
                }
                if (l1 > r0 || r1 < l0) bn = r1 - l1 + 1;
                else if (x1 >= x0) { bl = r0 + 1; bn = max(0, r1 - r0); }
                else bn = l0 - l1;
            }
            tc::cp_async_wait_all();
            __syncwarp();
            const int nr0 = b0 - t0 + 1, nc0 = r0 - l0 + 1, nc1 = r1 - l1 + 1;
            const int i0 = nr0 * ((nc0 + 3) >> 2), iA = i0 + an * ((nc1 + 3) >> 2), items = iA + in * ((bn + 3) >> 2);
            // item -> first position of its four candidates, how many there are, and its patch
            auto at_row = [&](const f32x2 *patch, int r) { return patch + (r & 1 ? odd : 0) + (r >> 1) * P; };
            auto decode = [&](int item, int &y, int &x, int &nv) -> const f32x2 * {
                if (item < i0) {
                    const int q = item / nr0;
                    y = t0 + item - q * nr0;
                    x = l0 + 4 * q;
                    nv = nc0 - 4 * q;
                    return at_row(patch0, y - t0) + (x - l0);
                }
                if (item < iA) {
                    const int e = item - i0, q = e / an;
                    y = at + e - q * an;
                    x = l1 + 4 * q;
                    nv = nc1 - 4 * q;
                } else {
                    const int e = item - iA, q = e / in;
                    y = it + e - q * in;
                    x = bl + 4 * q;
                    nv = bn - 4 * q;
                }
                return at_row(patch1, y - t1) + (x - l1);
            };
            LaneBest lb;
            lb.clear();
            int left = 0, nslots = 0;
            for (int base = 0; base < items; base += 32, nslots += 4) {
                const int item = base + lane;
                int y = 0, x = 0, nv = 0;
                const f32x2 *w0 = patch0;
                if (item < items) w0 = decode(item, y, x, nv);
                float acc[4][4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[u][k] = 0.0f;
                // pairs of rows: difference and square packed, then each row's columns k and 4 + k into lane sum k
#pragma unroll
                for (int yy = 0; yy < 4; ++yy) {
                    f32x2 w[11], r[8];
#pragma unroll
                    for (int k = 0; k < 11; ++k) w[k] = w0[yy * P + k];
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(rpair + yy * 8 + k);
                        r[k] = q.x;
                        r[k + 1] = q.y;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float lo[8], hi[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const f32x2 v = sub2(r[k], w[u + k]);
                            unpack2(mul2(v, v), lo[k], hi[k]);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[u][k] = __fadd_rn(__fadd_rn(acc[u][k], lo[k]), lo[4 + k]);
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc[u][k] = __fadd_rn(__fadd_rn(acc[u][k], hi[k]), hi[4 + k]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float d = lane_combine(acc[u]);
                    d = u < nv && dist_valid(d, a.thSSE) ? d : inf;
                    col[(nslots + u) * 32] = d;
                    left += d < inf;
                    lb.offer(d, nslots + u);
                }
            }
            float d, cut;
            int own, slot;
            int nf = warp_smallest(lb, col, nslots, left, G, d, own, slot, cut);
            const float key = lane < nf ? dist_to_key(d, a.distMul) : inf;
            const float prev = __shfl_up_sync(0xffffffffu, key, 1);
            const float last = __shfl_sync(0xffffffffu, key, G - 1);
            bool tie = lane >= 1 && lane < nf && !(prev < key);
            if (cut < inf) tie = tie || !(last < dist_to_key(cut, a.distMul));
            if (__any_sync(0xffffffffu, tie)) {
                // equal keys: the reference's heap order over the scan-ordered union decides
                if (lane == 0) { cen[0] = c0; cen[1] = c1; }
                nf = vbm_frame_general(a, rblk, plane, cen, ncen, work, fk, fp);
            } else if (lane < nf) {
                int y, x, nv;
                decode((slot >> 2) * 32 + own, y, x, nv);
                fk[lane] = key;
                fp[lane] = pack_yx(y, x + (slot & 3));
            }
            __syncwarp();
            for (int k = lane; k < nf; k += 32) {
                lp[L + k] = pack_zyx(fz, unpack_y(fp[k]), unpack_x(fp[k]));
                lk[L + k] = fk[k];
            }
            ncen = min(a.ps_num, nf);
            if (ncen > 0) c0 = fp[0];
            if (ncen > 1) c1 = fp[1];
            L += nf;
        }
    }
    __syncwarp();

    // final merge: partial_sort(begin + 1, begin + G) if longer than G
    uint32_t *op = a.out_pos + ob * G;
    float *ok = a.out_key ? a.out_key + ob * G : nullptr;
    if (L <= G) {
        for (int k = lane; k < L; k += 32) {
            op[k] = lp[k];
            if (ok) ok[k] = lk[k];
        }
        if (lane == 0) a.out_n[ob] = L;
        return;
    }
    const int K = G - 1;
    // the list's keys as lane columns (the work region holds list_cap values: 32 * slots)
    float *mcol = work + lane;
    LaneBest lb;
    lb.clear();
    int left = 0, nslots = 0;
    for (int c0 = 1; c0 < L; c0 += 32, ++nslots) {
        const float v = c0 + lane < L ? lk[c0 + lane] : inf;
        mcol[nslots * 32] = v;
        left += v < inf;
        lb.offer(v, nslots);
    }
    float d, cut;
    int own, slot;
    const int n = warp_smallest(lb, mcol, nslots, left, K, d, own, slot, cut);
    const float prev = __shfl_up_sync(0xffffffffu, d, 1);
    const float last = __shfl_sync(0xffffffffu, d, K - 1);
    const bool tie = (lane >= 1 && lane < n && !(prev < d)) || !(last < cut);
    if (!__any_sync(0xffffffffu, tie)) {
        if (lane < K) {
            op[1 + lane] = lp[1 + slot * 32 + own];
            if (ok) ok[1 + lane] = d;
        }
        if (lane == 0) {
            op[0] = lp[0];
            if (ok) ok[0] = lk[0];
            a.out_n[ob] = G;
        }
    } else if (lane == 0) {
        float *hk = fk;
        int *hi = reinterpret_cast<int *>(fp);
        for (int k = 0; k < K; ++k) { hk[k] = lk[1 + k]; hi[k] = 1 + k; }
        heap_make(hk, hi, K);
        for (int c = 1 + K; c < L; ++c) heap_offer(hk, hi, K, lk[c], c);
        heap_sort(hk, hi, K);
        op[0] = lp[0];
        if (ok) ok[0] = lk[0];
        for (int k = 0; k < K; ++k) {
            op[1 + k] = lp[hi[k]];
            if (ok) ok[1 + k] = hk[k];
        }
        a.out_n[ob] = G;
    }
}

}  // namespace bm3d
