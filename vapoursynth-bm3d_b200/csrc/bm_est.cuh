// bm_est.cuh -- K1 for 8 x 8 blocks, candidate step 1 and groups of at most 32: the full search with
// estimated distances, an error-bounded short list, and the exact distances of the short list.
//
// Same contract and output as bm_full_kernel (Block::BlockMatchingMulti, include/Block.h:554-729): the
// reference's distance is 64 separately rounded squares and sums per candidate, which no two reference
// blocks can share.  An estimate may: four neighbouring reference blocks of a row (at the profile's
// block step) have most of their pixels in common, so at one displacement the squared differences of
// their union, 8 + 3 * step columns, are summed once per column pair with fused multiply-adds, and each
// block's estimate is the sum of its columns.  Any order of 64 non-negative terms is within 64 * 2^-24 of
// their sum, relatively, and the reference's order is within 66 * 2^-24; so estimate and exact distance
// agree within kEstEps = 2^-16 (twice the sum of both), and a candidate whose estimate exceeds the bound
// on the K + 1 best by more than that is settled.
//
// The rest -- K + 1 candidates and the few within 2^-16 of the cut -- get exact distances and are
// sorted; when more than 64 remain, when too few are surely valid, or when kept keys or the cut are
// equal (the reference's tie order), the block is redone by bm_full_kernel's routines.
//
// Layout: four warps per CTA and four reference blocks (a team).  Their search windows, with the parts
// outside the plane left out, are staged in shared memory as pairs of rows, (0, 1) (2, 3) ... and again as
// (1, 2) (3, 4) ...: a candidate at any row and column then finds its pixels as aligned packed pairs
// (pairs of columns would have to be re-packed by moves for every other displacement, 75 moves per window row).
// Lane = displacement (W adjacent ones, rows of the window across the lanes); then one warp per block selects.
// Bound: the FP32 pipe in the estimates (2 operations a column instead of 3 a pixel and block).
// 1920x1080, range 16, 1,089 candidates, 8 frames: step 4, G 16: 13.1 ms exact, 6.7 ms here;
// step 3, G 32: 23.6 ms exact, 12.5 ms here.  (A form with tensor-core estimates in fp16, whose error bands sent a
// third of smooth pictures' candidates to the exact re-rank, took 10.0 and 21.5 ms.)
#pragma once

#include "bm.cuh"

namespace bm3d {

constexpr float kEstEps = 1.52587890625e-5f;    // 2^-16
constexpr int kEstCtas = 5;                     // CTAs per SM: 96 registers a thread, 41 KB at range 16
constexpr float kEstTiny = 1e-30f;              // below it a distance may round to zero (never a match)
// Largest threshold of this form.  A larger one is infinite in fp32, or nearly: then an infinite distance is a
// match, which the empty slots of the estimates could not be told from, and the exact search takes the call.
constexpr float kEstMaxThr = 1e38f;

__device__ __forceinline__ f32x2 fma2_(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The union of four blocks at step S is cut at their edges into segments that no edge crosses: segment of
// column x (and the number of segments, at x = NC)
__host__ __device__ constexpr int est_segment(int S, int x)
{
    int c = 0;
    for (int b = 1; b <= x; ++b) {
        bool edge = false;
        for (int n = 0; n < 4; ++n) edge = edge || b == n * S || b == n * S + 8;
        c += edge;
    }
    return c;
}

// Squared-difference sums of the W displacements that start at `w0` (row pairs, pitch P) against the four
// blocks of the strip rs (row pairs, RS columns): est[d][n] of block n
template <int S, int W, int RS>
__device__ __forceinline__ void strip_estimates(const f32x2 *w0, int P, const f32x2 *rs, float (&est)[W][4])
{
    constexpr int NC = 8 + 3 * S, NS = est_segment(S, NC - 1) + 1;
    f32x2 acc[W][NS];
#pragma unroll
    for (int d = 0; d < W; ++d)
#pragma unroll
        for (int k = 0; k < NS; ++k) acc[d][k] = 0ull;
#pragma unroll 1
    for (int y = 0; y < 4; ++y) {
        f32x2 w[W];
#pragma unroll
        for (int d = 0; d < W - 1; ++d) w[d] = w0[y * P + d];
#pragma unroll
        for (int x = 0; x < NC; x += 2) {
            const ulonglong2 r2 = *reinterpret_cast<const ulonglong2 *>(rs + y * RS + x);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (x + h >= NC) break;
                w[(x + h + W - 1) % W] = w0[y * P + x + h + W - 1];
                const f32x2 r = h ? r2.y : r2.x;
#pragma unroll
                for (int d = 0; d < W; ++d) {
                    const f32x2 v = sub2(r, w[(x + h + d) % W]);
                    acc[d][est_segment(S, x + h)] = fma2_(v, v, acc[d][est_segment(S, x + h)]);
                }
            }
        }
    }
#pragma unroll
    for (int d = 0; d < W; ++d) {
        float s[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            float lo, hi;
            unpack2(acc[d][k], lo, hi);
            s[k] = lo + hi;
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            float e = s[est_segment(S, n * S)];
#pragma unroll
            for (int k = est_segment(S, n * S) + 1; k <= est_segment(S, n * S + 7); ++k) e += s[k];
            est[d][n] = e;
        }
    }
}

// Exact distance (the reference's order) of two 8 x 8 blocks held as row pairs: four lane sums, lane k taking
// columns k and 4 + k of every row
__device__ __forceinline__ float exact_pairs(const f32x2 *r, int rp, const f32x2 *w, int wp)
{
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        float lo[8], hi[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const f32x2 d = sub2(r[y * rp + x], w[y * wp + x]);
            unpack2(mul2(d, d), lo[x], hi[x]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = __fadd_rn(__fadd_rn(acc[k], lo[k]), lo[4 + k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = __fadd_rn(__fadd_rn(acc[k], hi[k]), hi[4 + k]);
    }
    return lane_combine(acc);
}

template <int S, int W>
__global__ void __launch_bounds__(128, kEstCtas) bm_est_kernel(BMArgs a, EstLayout L)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int NC = 8 + 3 * S, RS = (NC + 1) & ~1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int f = blockIdx.z, by = blockIdx.y;
    const int R = a.range, span = 2 * R + 1, nlat = span * span, P = L.pitch;
    const float *plane = a.ref + (long long)f * a.frame_stride;
    const float inf = __int_as_float(0x7f800000);
    // the strip of the team's blocks, block (0, 0), the window as pairs of rows from an even and from an odd one
    f32x2 *rs = reinterpret_cast<f32x2 *>(smem), *zero = rs + 4 * RS, *even = zero + 32, *odd = even + L.odd;
    float *sdall = reinterpret_cast<float *>(even + L.cells);

    // the team: blocks at xf + n * S; the last block of a row, where it is off that grid, is a team of its
    // own.  Positions of the scan: multiples of the step, the last ones moved inside the plane.
    const bool tail = (int)blockIdx.x >= L.teams;
    const int bx0 = tail ? a.nbx - 1 : 4 * (int)blockIdx.x;
    const int nref = tail ? 1 : min(4, L.nreg - bx0);
    const int j = min(by * S, a.H - 8), xf = min(bx0 * S, a.W - 8);

    // the block at (0, 0), two pixels per lane
    const float o0 = __ldg(plane + (long long)(lane >> 3) * a.ld + (lane & 7));
    const float o1 = __ldg(plane + (long long)((lane >> 3) + 4) * a.ld + (lane & 7));
    // window rows j - R .. j + R + 7, columns xf - R .. xf + R + NC - 1 in 16-byte chunks, as far as the
    // chunks lie in the plane's rows (ld is a multiple of 4); window column xo is plane column xf - R.  The
    // strip of the reference blocks on the way.
    const int xw = (xf - R) & ~3, xo = xf - R - xw;
    const int qn = (xo + 2 * R + NC + 3) >> 2;
    for (int q = tid & 15; q < qn; q += 16) {
        const int x = xw + 4 * q, xr = 4 * q - xo - R;        // plane column, strip column
        if (x < 0 || x >= a.ld) continue;
        const float *src = plane + x;
        for (int r0 = tid >> 4; r0 < 2 * R + 8; r0 += 5 * 8) {
            float4 v[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int y = j - R + r0 + 8 * k;
                if (r0 + 8 * k < 2 * R + 8 && y >= 0 && y < a.H) v[k] = __ldg(reinterpret_cast<const float4 *>(src + (long long)y * a.ld));
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int r = r0 + 8 * k;
                if (r >= 2 * R + 8 || j - R + r < 0 || j - R + r >= a.H) continue;
                const float p[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                // word r & 1 of the pair from an even row, the other word of the pair from an odd one
                float *e = reinterpret_cast<float *>(even + (r >> 1) * P + 4 * q) + (r & 1);
                float *o = reinterpret_cast<float *>(odd + ((r + 1) / 2 - 1) * P + 4 * q) + 1 - (r & 1);
#pragma unroll
                for (int m = 0; m < 4; ++m) e[2 * m] = p[m];
                if (r > 0 && r < 2 * R + 7) {
#pragma unroll
                    for (int m = 0; m < 4; ++m) o[2 * m] = p[m];
                }
                if (r >= R && r < R + 8 && xr > -4 && xr < RS) {
                    float *t = reinterpret_cast<float *>(rs + ((r - R) >> 1) * RS + xr) + ((r - R) & 1);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (xr + m >= 0 && xr + m < RS) t[2 * m] = p[m];
                }
            }
        }
    }
    if (warp == 0) {
        float *z = reinterpret_cast<float *>(zero + (lane >> 4) * 8 + (lane & 7)) + ((lane >> 3) & 1);
        z[0] = o0;
        z[32] = o1;
    }
    __syncthreads();

    // estimates of every displacement; candidates outside the plane and at distance zero (the block
    // itself) are left out (infinite)
    const int nq = (span + W - 1) / W;
    // the window from row r on, as pairs of rows
    auto rowpair = [&](int r) { return (r & 1 ? odd : even) + (r >> 1) * P; };
    const float thsure = a.thSSE * (1.0f + kEstEps);
    const bool inside = j >= R && j + R <= a.H - 8 && xf >= R && xf + 3 * S + R <= a.W - 8;
    for (int it = tid; it < nq * span; it += 128) {
        const int q = (int)(((float)it + 0.5f) * (1.0f / (float)span)), ry = it - q * span;
        const int y = j - R + ry;
        const bool iny = y >= 0 && y <= a.H - 8;
        float est[W][4];
        strip_estimates<S, W, RS>(rowpair(ry) + xo + W * q, P, rs, est);
        float *o = sdall + ry * span + W * q;
#pragma unroll
        for (int d = 0; d < W; ++d) {
            if (W * q + d >= span) break;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                bool in = est[d][n] > 0.0f;
                if (!inside) {
                    const int x = xf + n * S - R + W * q + d;
                    in = in && iny && x >= 0 && x <= a.W - 8;
                }
                o[n * L.cs + d] = in ? est[d][n] : inf;
            }
        }
    }
    // the trailing (0, 0) candidate (block `warp`), then infinite padding
    float *sd = sdall + warp * L.cs;
    {
        const float *t = reinterpret_cast<const float *>(rs + (lane >> 4) * RS + warp * S + (lane & 7)) + ((lane >> 3) & 1);
        const float d0 = t[0] - o0, d1 = t[4 * RS] - o1;
        float s = fmaf(d0, d0, d1 * d1);
        s = warp_sum(s);
        if (lane == 0) sd[nlat] = s > 0.0f ? s : inf;
        for (int c = nlat + 1 + lane; c < L.cs; c += 32) sd[c] = inf;
    }
    __syncthreads();
    if (warp >= nref) return;

    // ---- selection, one warp per block --------------------------------------------------------------
    const int n = warp, i = xf + n * S;
    const int G = a.G, K = G - 1;
    uint32_t *list = reinterpret_cast<uint32_t *>(sdall + 4 * L.cs) + n * 320;
    float *dl = reinterpret_cast<float *>(list + 64), *ks = dl + 64;
    const size_t ob = ((size_t)f * a.nby + by) * a.nbx + bx0 + n;
    const uint32_t ref_pos = pack_yx(j, i);
    uint32_t *opos = a.out_pos + ob * G;
    float *okey = a.out_key ? a.out_key + ob * G : nullptr;

    // The threshold is finite with its margin (kEstMaxThr), so an empty slot, which is infinite, passes no test
    // below.  The K + 1 smallest estimates among the surely valid, out of each lane's two smallest: an upper
    // bound on the K + 1 smallest distances.  Lane l takes element (l + 7 k) mod 32 of round k, so
    // that a compact patch of good candidates is spread over the lanes.
    const float ths = a.thSSE * (1.0f - 2.0f * kEstEps);
    float f1 = inf, f2 = inf;
    int nsure = 0;
    const int rounds = L.cs >> 5;
#pragma unroll 5
    for (int k = 0; k < rounds; ++k) {
        const float v = sd[32 * k + ((lane + 7 * k) & 31)];
        const bool sure = v <= ths && v >= kEstTiny;
        nsure += sure;
        const float h = sure ? v : inf;
        f2 = fminf(f2, fmaxf(f1, h));
        f1 = fminf(f1, h);
    }
    nsure = warp_sum(nsure);
    bool done = false;
    // complete: every candidate that may be valid is listed
    const bool complete = nsure <= K;
    float cut = inf;
    if (!complete) {
        float v2[2] = {f1, f2};
        warp_bitonic_f32<2>(v2);
        cut = __shfl_sync(0xffffffffu, v2[0], K);
    }
    const float bnd = fminf(a.thSSE, cut * (1.0f + 2.0f * kEstEps));      // on the exact distances
    const float bt = fminf(thsure, cut * (1.0f + 4.0f * kEstEps));        // on the estimates
    // the band: every lane's own hits (at most kHits are kept), then one after the other
    constexpr int kHits = 8;
    int cnt = 0;
    uint32_t *mine = list + 64 + lane;
#pragma unroll 5
    for (int k = 0; k < rounds; ++k) {
        const int c = 32 * k + ((lane + 7 * k) & 31);
        const bool hit = sd[c] <= bt;
        if (hit) mine[32 * min(cnt, kHits - 1)] = (uint32_t)c;
        cnt += hit;
    }
    int ms = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, ms, o);
        if (lane >= o) ms += v;
    }
    const int at = ms - cnt;
    ms = __shfl_sync(0xffffffffu, ms, 31);
    const bool fits = ms <= 64 && __all_sync(0xffffffffu, cnt <= kHits);
    if (fits)
        for (int k = 0; k < cnt; ++k) list[at + k] = mine[32 * k];
    __syncwarp();
    // c / span: exact for c below 2^15 (the rounding error is far below half a step of the quotient)
    const float rspan = 1.0f / (float)span;
    auto row_of = [=](int c) { return (int)(((float)c + 0.5f) * rspan); };
    auto pos_of = [=](uint32_t c) -> uint32_t {
        const int ry = row_of((int)c), cc = (int)c - ry * span;
        return (int)c >= nlat ? pack_yx(0, 0) : pack_yx(j - R + ry, i - R + cc);
    };
    if (fits) {
        // exact distances in the reference's order, four lanes per candidate: lane k of a quad takes its
        // k-th partial sum (columns k and 4 + k of every row)
        const int k4 = lane & 3;
        float rb[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) rb[e] = reinterpret_cast<const float *>(rs + (e >> 2) * RS + n * S + 4 * (e & 1) + k4)[(e >> 1) & 1];
        float nd[2] = {inf, inf};              // distances of list entries lane and lane + 32
        for (int e = 0; 8 * e < ms; ++e) {
            const int idx = 8 * e + (lane >> 2);
            const int c = idx < ms ? (int)list[idx] : 0;
            const int ry = row_of(c), cc = c - ry * span;
            const bool org = c >= nlat;
            const float *w = reinterpret_cast<const float *>(org ? zero + k4 : rowpair(ry) + xo + n * S + cc + k4);
            const int ws = 2 * (org ? 8 : P);
            float s = 0.0f;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                const float d = __fsub_rn(rb[m], w[(m >> 2) * ws + 8 * (m & 1) + ((m >> 1) & 1)]);
                s = __fadd_rn(s, __fmul_rn(d, d));
            }
            const float s0 = __shfl_sync(0xffffffffu, s, 0, 4), s1 = __shfl_sync(0xffffffffu, s, 1, 4);
            const float s2 = __shfl_sync(0xffffffffu, s, 2, 4), s3 = __shfl_sync(0xffffffffu, s, 3, 4);
            float d = __fadd_rn(__fadd_rn(__fadd_rn(s0, s1), s2), s3);
            d = idx < ms && dist_valid(d, a.thSSE) ? d : inf;
            d = __shfl_sync(0xffffffffu, d, 4 * (lane & 7));
            if ((lane >> 3) == (e & 3)) {
                if (e < 4) nd[0] = d;
                else nd[1] = d;
            }
        }
        dl[lane] = nd[0];
        dl[lane + 32] = nd[1];
        ks[lane] = __int_as_float(0x7fc00000);      // NaN: a rank that no entry takes
        const int nval = warp_sum((int)(nd[0] < inf) + (int)(nd[1] < inf));
        const int nbelow = warp_sum((int)(nd[0] <= bnd) + (int)(nd[1] <= bnd));
        __syncwarp();
        // complete: the band holds every valid candidate.  Else it holds at least K + 1 at or below
        // bnd and everything outside lies above bnd, so its first K + 1 are the first K + 1 of all
        // (the last one tells whether the cut falls between equal keys).
        if (complete || nbelow > K) {
            // rank of the lane's entries; equal distances share a rank and leave another without an entry
            int r0 = 0, r1 = 0;
            for (int e = 0; e < ms; e += 4) {
                const float4 q = *reinterpret_cast<const float4 *>(dl + e);
                r0 += (q.x < nd[0]) + (q.y < nd[0]) + (q.z < nd[0]) + (q.w < nd[0]);
                r1 += (q.x < nd[1]) + (q.y < nd[1]) + (q.z < nd[1]) + (q.w < nd[1]);
            }
            const int nout = min(nval, K), last = min(nval - 1, K);     // ranks 0 .. last must have rising keys
            const float k0 = dist_to_key(nd[0], a.distMul), k1 = dist_to_key(nd[1], a.distMul);
            if (nd[0] < inf && r0 < 32) ks[r0] = k0;
            if (nd[1] < inf && r1 < 32) ks[r1] = k1;
            __syncwarp();
            const bool bad = lane <= last && !(lane ? ks[lane - 1] < ks[lane] : ks[0] >= 0.0f);
            if (!__any_sync(0xffffffffu, bad)) {
                if (lane == 0) {
                    opos[0] = ref_pos;
                    if (okey) okey[0] = 0.0f;
                    a.out_n[ob] = 1 + nout;
                }
                if (nd[0] < inf && r0 < nout) {
                    opos[1 + r0] = pos_of(list[lane]);
                    if (okey) okey[1 + r0] = k0;
                }
                if (nd[1] < inf && r1 < nout) {
                    opos[1 + r1] = pos_of(list[lane + 32]);
                    if (okey) okey[1 + r1] = k1;
                }
                done = true;
            }
        }
    }
    __syncwarp();
    if (!done) {
        // every exact distance over the clipped lattice, then the plain selection
        if (lane == 0 && a.stats) atomicAdd(a.stats + 1, 1ull);
        const int t = max(0, j - R), b = min(a.H - 8, j + R), l = max(0, i - R), r = min(a.W - 8, i + R);
        const int nrows = b - t + 1, ncols = r - l + 1, clat = nrows * ncols;
        for (int c = lane; c <= clat; c += 32) {
            const int ry = c / ncols, cc = c - ry * ncols;
            const bool org = c == clat;
            sd[c] = exact_pairs(rs + n * S, RS, org ? zero : rowpair(t + ry - j + R) + xo + l + cc - xf + R, org ? 8 : P);
        }
        __syncwarp();
        auto pos_clip = [=](uint32_t c) -> uint32_t {
            if ((int)c >= clat) return pack_yx(0, 0);
            const int ry = (int)c / ncols, cc = (int)c - ry * ncols;
            return pack_yx(t + ry, l + cc);
        };
        float *hk = reinterpret_cast<float *>(list + 64);
        select_and_emit(sd, clat + 1, list, hk, reinterpret_cast<int *>(hk + 32), a, ref_pos, ob, pos_clip);
    }
}

}  // namespace bm3d
