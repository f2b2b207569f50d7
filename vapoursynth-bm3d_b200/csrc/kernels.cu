// kernels.cu -- the single CUDA translation unit holding every sm_100a kernel of the library
// (block matching, predictive search, collaborative filter, conversions) and their launchers.

#include "common.cuh"
#include "select.cuh"
#include "bm.cuh"
#include "bm_est.cuh"
#include "proposal.cuh"
#include "vbm.cuh"
#include "cf.cuh"
#include "cf_box.cuh"
#include "cf_mid.cuh"
#include "cf_tc.cuh"
#include "fp64.cuh"
#include "convert.cuh"
#include "launch.h"
#include "params.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

namespace bm3d {

// Every kernel launch of the library goes through a launcher below and is counted here.
static std::atomic<unsigned long long> g_launches{0};
unsigned long long launch_count() { return g_launches.load(); }
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
#define COUNT_LAUNCH() g_launches.fetch_add(1, std::memory_order_relaxed)

template <typename K>
static cudaError_t allow_smem(K kernel, size_t bytes)
{
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// ---- learned proposal ----------------------------------------------------------------------------

int prop_triplet_bytes() { return (int)sizeof(PropTriplet); }

cudaError_t launch_prop_features(const float *x, int ld, int W, int H, const float *wt, void *hid, void *feat, float *rs,
                                 void *desc, cudaStream_t s)
{
    if (W < 8 || H < 8) return cudaErrorInvalidValue;
    auto *h = static_cast<__nv_bfloat16 *>(hid);
    auto *f = static_cast<__nv_bfloat16 *>(feat);
    const dim3 blk(128);
    COUNT_LAUNCH();
    prop_conv1_kernel<<<dim3((W + 127) / 128, H), blk, 0, s>>>(x, ld, W, H, wt, h);
    COUNT_LAUNCH();
    prop_conv2_kernel<<<dim3((W + 128 * kPropConv2Px - 1) / (128 * kPropConv2Px), H), blk, 0, s>>>(h, W, H, wt, f);
    COUNT_LAUNCH();
    prop_rowsum_kernel<<<dim3((W - 3 + 127) / 128, H, kPropCh), blk, 0, s>>>(f, W, H, rs);
    COUNT_LAUNCH();
    prop_desc_kernel<<<dim3((W - 7 + 127) / 128, H - 7), blk, 0, s>>>(rs, W, H, static_cast<__nv_bfloat16 *>(desc));
    return cudaGetLastError();
}

cudaError_t launch_prop_loss(const void *triplets, int ntr, const void *desc, long long dstride, int Wd, float *gD,
                             float scale, float *loss, cudaStream_t s)
{
    COUNT_LAUNCH();
    prop_rank_loss_kernel<<<(ntr + 127) / 128, 128, 0, s>>>(static_cast<const PropTriplet *>(triplets), ntr,
                                                           static_cast<const __nv_bfloat16 *>(desc), dstride, Wd, gD, scale, loss);
    return cudaGetLastError();
}

cudaError_t launch_prop_backward(const float *x, int ld, int W, int H, const float *wt, const void *hid, const float *gD,
                                 float *dF, float *dH, float *gw, cudaStream_t s)
{
    const dim3 blk(128), grd((W + 127) / 128, H);
    COUNT_LAUNCH();
    prop_desc_bwd_kernel<<<grd, blk, 0, s>>>(gD, W, H, dF);
    COUNT_LAUNCH();
    prop_conv2_bwd_kernel<<<grd, blk, 0, s>>>(static_cast<const __nv_bfloat16 *>(hid), dF, W, H, wt, gw, dH);
    COUNT_LAUNCH();
    prop_conv1_bwd_kernel<<<grd, blk, 0, s>>>(x, ld, dH, W, H, gw);
    return cudaGetLastError();
}

cudaError_t launch_prop_adam(float *wt, const float *g, float *m, float *v, float lr, float b1t, float b2t, cudaStream_t s)
{
    COUNT_LAUNCH();
    prop_adam_kernel<<<(kPropWeights + 255) / 256, 256, 0, s>>>(wt, g, m, v, lr, b1t, b2t);
    return cudaGetLastError();
}

cudaError_t launch_prop_sample(const float *frames, long long fstride, int ld, int W, int H, int nframes, const uint32_t *lists,
                               const int *counts, int G, const int *sy, const int *sx, int nby, int nbx, int range,
                               uint32_t seed, void *out, int ntr, cudaStream_t s)
{
    COUNT_LAUNCH();
    prop_sample_kernel<<<(ntr + 127) / 128, 128, 0, s>>>(frames, fstride, ld, W, H, nframes, lists, counts, G, sy, sx, nby,
                                                        nbx, range, seed, static_cast<PropTriplet *>(out), ntr);
    return cudaGetLastError();
}

cudaError_t launch_bm_learned(const BMArgs &a, const void *desc, int nprop, int nframes, size_t smem, cudaStream_t s)
{
    if (a.B != 8 || a.G > 32) return cudaErrorInvalidValue;
    dim3 grid((a.nbx + a.warps - 1) / a.warps, a.nby, nframes);
    cudaError_t e;
    if ((e = allow_smem(bm_learned_kernel, smem)) != cudaSuccess) return e;
    COUNT_LAUNCH();
    bm_learned_kernel<<<grid, 32 * a.warps, smem, s>>>(a, static_cast<const __nv_bfloat16 *>(desc), nprop);
    return cudaGetLastError();
}

template <int S, int W>
static cudaError_t launch_bm_est_t(const BMArgs &a, const EstLayout &L, int nframes, cudaStream_t s)
{
    cudaError_t e;
    if ((e = allow_smem(bm_est_kernel<S, W>, L.bytes)) != cudaSuccess) return e;
    COUNT_LAUNCH();
    bm_est_kernel<S, W><<<dim3(L.teams + (L.nreg < a.nbx), a.nby, nframes), 128, L.bytes, s>>>(a, L);
    return cudaGetLastError();
}

int launch_bm_est(const BMArgs &a, int block_step, int last, int nframes, cudaStream_t s, cudaError_t *e)
{
    if (a.B != 8 || a.step != 1 || a.G < 2 || a.G > 32 || block_step > kEstMaxStep || !(a.thSSE <= kEstMaxThr)) return 0;
    // displacements per lane: 3 or 4, whichever leaves fewer slots of the team's 128 lanes unused
    const int span = 2 * a.range + 1;
    if (span * span >= 1 << 15) return 0;
    auto slots = [span](int W) { return ((span + W - 1) / W * span + 127) / 128 * W; };
    const int W = slots(4) < slots(3) ? 4 : 3;
    const EstLayout L = est_layout(a.range, block_step, W, a.nbx, last);
    if (L.bytes > 200 * 1024) return 0;
    switch (block_step * 8 + W) {
#define BM3D_EST(S) \
    case S * 8 + 3: *e = launch_bm_est_t<S, 3>(a, L, nframes, s); return 1; \
    case S * 8 + 4: *e = launch_bm_est_t<S, 4>(a, L, nframes, s); return 1;
    BM3D_EST(1) BM3D_EST(2) BM3D_EST(3) BM3D_EST(4) BM3D_EST(5) BM3D_EST(6) BM3D_EST(7) BM3D_EST(8)
#undef BM3D_EST
    default: return 0;
    }
}

cudaError_t launch_bm_full(const BMArgs &a, int nframes, size_t smem, cudaStream_t s)
{
    dim3 grid((a.nbx + a.warps - 1) / a.warps, a.nby, nframes);
    dim3 block(32 * a.warps);
    cudaError_t e;
    if (a.B == 8) {
        if ((e = allow_smem(bm_full_kernel<8>, smem)) != cudaSuccess) return e;
        COUNT_LAUNCH();
        bm_full_kernel<8><<<grid, block, smem, s>>>(a);
    } else {
        if ((e = allow_smem(bm_full_kernel<0>, smem)) != cudaSuccess) return e;
        COUNT_LAUNCH();
        bm_full_kernel<0><<<grid, block, smem, s>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_vbm_predict(const VBMArgs &a, bool fast, int nframes, size_t smem, cudaStream_t s)
{
    dim3 grid((a.nbx + a.warps - 1) / a.warps, a.nby, nframes);
    dim3 block(32 * a.warps);
    cudaError_t e;
    if (fast) {
        if ((e = allow_smem(vbm_predict8_kernel, smem)) != cudaSuccess) return e;
        COUNT_LAUNCH();
        vbm_predict8_kernel<<<grid, block, smem, s>>>(a);
        return cudaGetLastError();
    }
    if ((e = allow_smem(vbm_predict_kernel, smem)) != cudaSuccess) return e;
    COUNT_LAUNCH();
    vbm_predict_kernel<<<grid, block, smem, s>>>(a);
    return cudaGetLastError();
}

int cf_fast_supported(int B, int G) { return B == 8 && (G == 8 || G == 16 || G == 32); }

// Two CTAs of four warp pairs per SM: shared memory of one, and how many run at once
constexpr int kBoxPairs = 4, kBoxCap = 115712, kBoxResident = 2 * 148;

// Tile of reference blocks for cf_box_kernel / cf_boxh_kernel; fills the geometry and returns whether the box form is the
// one to take.  A pair takes one slot of 32 / G groups per step (Basic: two), and staging and flushing the box cost about
// half a step: the tile with the least waves x (steps + 1/2) is taken (so that a small frame gets small tiles and
// all SMs; 352x288 at profile fast, 1,584 groups: 34 us with the largest tile, 30 us).
// launch_cf_pair takes the others:
// - Where no tile that fits fills three quarters of a step, pairs idle and a box is staged for a few groups.
//   1920x1080 YUV x 3, box and pairs: Basic, range 24, step 4, G = 16 (one slot of eight) 20.2 and 3.5 ms; range 20 (six
//   of eight) 4.9 and 3.5 ms, still ahead of a warp per group (5.4 ms); Final, range 20, step 4, G = 16 (one of four) 15.1
//   and 5.2 ms.  (Three CTAs of two pairs, or one of four in all shared memory, gain nothing on the pairs at any range:
//   Final, range 36, step 8, G = 8: 2.47 and 0.70 ms.)
// - Where a window has fewer than 4 G candidates, most lists are short and of any length, and the slow direct
//   sums of one pair hold up its CTA's tile.  640x480, step 3: Basic, G = 16, range 3 184 and 141 us, range 4 143 and
//   137 us; Final, G = 32, range 5 794 and 489 us, range 6 485 and 515 us.
static bool cf_box_fit(const CFArgs &a, CFBox &g, int step, int G, size_t *smem)
{
    const int gpw = 32 / G;
    const int cell = a.wiener ? 16 : 12, per_step = a.wiener ? kBoxPairs : 2 * kBoxPairs;   // bytes of a cell, slots of a step
    const int span = 2 * g.range + 1;
    if (span * span < 4 * G) return false;
    double best = 0.0;
    int most = 0;                                            // slots of the largest tile
    for (int ny = 1; ny <= 8; ++ny)
        for (int nx = gpw; nx * ny <= 128; nx += gpw) {
            const int w = (2 * g.range + 8 + (nx - 1) * step + 3 + 3) & ~3;
            const int rows = std::min(a.H, 2 * g.range + 8 + (ny - 1) * step);
            const int pitch = w + ((12 - (w & 7)) & 7);      // 4 mod 8: a scatter step's eight rows in distinct banks
            const size_t bytes = (size_t)kBoxPairs * 32 * kBT * 8 + ((size_t)rows * pitch + 64) * cell +
                                 (size_t)kBoxPairs * 2 * gpw * 4 + (a.wiener ? 0 : (size_t)kBoxPairs * 2 * 4);
            if (bytes > kBoxCap) break;
            const int slots = ny * (nx / gpw), steps = (slots + per_step - 1) / per_step;
            most = std::max(most, slots);
            const int tx = (g.nbx + nx - 1) / nx, ty = (g.nby + ny - 1) / ny;
            double waves = (double)tx * ty * g.nplanes * (double)(a.ngroups / a.blocks_per_frame) / kBoxResident;
            if (waves < 6.0) waves = std::ceil(waves);
            const double cost = waves * (steps + 0.5);
            if (best > 0.0 && cost >= best) continue;
            best = cost;
            g.tx = tx;
            g.ty = ty;
            g.rows = rows;
            g.pitch = pitch;
            *smem = bytes;
        }
    return 4 * most >= 3 * per_step;
}

template <int G>
static int launch_cf_box_t(const CFArgs &a, CFBox g, int step, cudaStream_t s, cudaError_t *e)
{
    size_t smem = 0;
    if (!cf_box_fit(a, g, step, G, &smem)) return 0;
    auto kernel = a.wiener ? cf_box_kernel<G, kBoxPairs> : cf_boxh_kernel<G, kBoxPairs>;
    if ((*e = allow_smem(kernel, smem)) != cudaSuccess) return 1;
    const long long frames = a.ngroups / a.blocks_per_frame;
    COUNT_LAUNCH();
    kernel<<<dim3((unsigned)(frames * g.tx * g.ty), g.nplanes), kBoxPairs * 64, smem, s>>>(a, g);
    *e = cudaGetLastError();
    return 1;
}

int launch_cf_box(const CFArgs &a, const CFBox &g, int step, cudaStream_t s, cudaError_t *e)
{
    if (a.B != 8 || a.vbm3d) return 0;
    switch (a.G) {
    case 8: return launch_cf_box_t<8>(a, g, step, s, e);
    case 16: return launch_cf_box_t<16>(a, g, step, s, e);
    case 32: return launch_cf_box_t<32>(a, g, step, s, e);
    default: return 0;
    }
}

template <int G>
static cudaError_t launch_cf_pair_t(const CFArgs &a, cudaStream_t s)
{
    constexpr int NP = 4;
    auto kernel = a.wiener ? cf_pair_kernel<G, NP> : cf_pairh_kernel<G, NP>;
    const size_t smem = (size_t)NP * 32 * kBT * 8 + (size_t)NP * 2 * (32 / G) * 4;
    cudaError_t e;
    if ((e = allow_smem(kernel, smem)) != cudaSuccess) return e;
    const long long per = (long long)NP * (32 / G) * (a.wiener ? 1 : 2);       // groups of a CTA's step
    COUNT_LAUNCH();
    kernel<<<(unsigned)std::max<long long>(1, std::min<long long>((a.ngroups + per - 1) / per, 148LL * 8)), NP * 64, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_cf_pair(const CFArgs &a, cudaStream_t s)
{
    switch (a.B == 8 ? a.G : 0) {
    case 8: return launch_cf_pair_t<8>(a, s);
    case 16: return launch_cf_pair_t<16>(a, s);
    case 32: return launch_cf_pair_t<32>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int G, bool W>
static cudaError_t launch_cf_fast_t(const CFArgs &a, cudaStream_t s)
{
    cudaError_t e;
    // per-lane kernel: 4 warps per CTA, grid-stride over the groups
    const int warps = 4;
    const long long warps_needed = (a.ngroups + (32 / G) - 1) / (32 / G);
    const int grid = (int)std::max<long long>(1, std::min<long long>((warps_needed + warps - 1) / warps, 148LL * 64));
    const size_t smem = (size_t)warps * (W ? 2 : 1) * 32 * kTP * sizeof(float);
    if ((e = allow_smem(cf_fast_kernel<G, W>, smem)) != cudaSuccess) return e;
    COUNT_LAUNCH();
    cf_fast_kernel<G, W><<<grid, 32 * warps, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_cf_partial_list(const int *count, long long ngroups, int G, long long *list, unsigned int *n, cudaStream_t s)
{
    const long long blocks = std::max<long long>(1, std::min<long long>((ngroups + 255) / 256, 148LL * 16));
    COUNT_LAUNCH();
    cf_partial_list_kernel<<<(unsigned)blocks, 256, 0, s>>>(count, ngroups, G, list, n);
    return cudaGetLastError();
}

cudaError_t launch_cf_fast(const CFArgs &a, cudaStream_t s)
{
    if (a.B != 8) return cudaErrorInvalidValue;
    const bool w = a.wiener != 0;
    switch (a.G) {
    case 8: return w ? launch_cf_fast_t<8, true>(a, s) : launch_cf_fast_t<8, false>(a, s);
    // Wiener: only the short groups that the tensor-core kernel leaves, which takes all of these lengths
    case 16: return w ? cudaErrorInvalidValue : launch_cf_fast_t<16, false>(a, s);
    case 32: return w ? cudaErrorInvalidValue : launch_cf_fast_t<32, false>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

// ---- precision form: tensor-core collaborative filter ------------------------------------------

int cf_tc_supported(int B, int G) { return B == 8 && (G == 8 || G == 16 || G == 32); }

// tf32 value of x, rounded to nearest (ties away), as the tensor cores read it
static float round_tf32(float x)
{
    uint32_t u;
    std::memcpy(&u, &x, 4);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
    float r;
    std::memcpy(&r, &u, 4);
    return r;
}

template <int G>
static void tc_tables_t(std::vector<unsigned char> &img)
{
    using Lay = TcLayout<G>;
    img.assign(Lay::kTableBytes, 0);
    auto put = [&](uint32_t off, double v) {
        const float f = round_tf32((float)v);
        std::memcpy(img.data() + off, &f, 4);
    };
    // REDFT10 C[k][j] = 2 cos(pi (j + 1/2) k / N); REDFT01 Ci[j][k] = k == 0 ? 1 : 2 cos(pi k (j + 1/2) / N)
    auto fwd = [](int N, int k, int j) { return (double)cos2((long)(2 * j + 1) * k, 2L * N); };
    auto inv = [](int N, int j, int k) { return k == 0 ? 1.0 : (double)cos2((long)k * (2 * j + 1), 2L * N); };
    for (int w = 0; w < 128 / G; ++w)        // one copy of the matrices per group of a tile
        for (int kz = 0; kz < G; ++kz)
            for (int jz = 0; jz < G; ++jz) {
                put(Lay::kZf + tc_kmajor(G * w + kz, jz, G), fwd(G, kz, jz));
                put(Lay::kZi + tc_kmajor(G * w + jz, kz, G), inv(G, jz, kz));
            }
    for (int ky = 0; ky < 8; ++ky)
        for (int kx = 0; kx < 8; ++kx)
            for (int y = 0; y < 8; ++y)
                for (int x = 0; x < 8; ++x) {
                    const int c = ky * 8 + kx, px = y * 8 + x;
                    put(Lay::kKf + tc_kmajor(c, px, 64), fwd(8, ky, y) * fwd(8, kx, x));
                    put(Lay::kKi + tc_kmajor(px, c, 64), inv(8, y, ky) * inv(8, x, kx));
                }
}

// Rows of the n-point z-stage matrices, n = 1 .. G, as the Wiener kernels load them into tensor
// memory for tiles with a short group: [n - 1][forward, inverse][row j][G], forward row j = the
// REDFT10 coefficients of frequency j, inverse row j = the REDFT01 coefficients of block j, zero
// past n (rows and columns).
void cf_tc_partial_tables(int G, std::vector<float> &out)
{
    out.assign((size_t)G * 2 * G * G, 0.0f);
    for (int n = 1; n <= G; ++n)
        for (int r = 0; r < n; ++r)
            for (int k = 0; k < n; ++k) {
                float *f = out.data() + (size_t)(n - 1) * 2 * G * G;
                f[r * G + k] = round_tf32((float)cos2((long)(2 * k + 1) * r, 2L * n));
                f[G * G + r * G + k] = round_tf32(k == 0 ? 1.0f : (float)cos2((long)k * (2 * r + 1), 2L * n));
            }
}

int cf_tc_handles_partial(int B, int G, int wiener)
{
    if (!cf_tc_supported(B, G) || !wiener) return 0;
    return G == 16 ? TcShape<16, true>::kShort : G == 32 ? TcShape<32, true>::kShort : TcShape<8, true>::kShort;
}

void cf_tc_tables(int G, std::vector<unsigned char> &img)
{
    if (G == 8) tc_tables_t<8>(img);
    else if (G == 16) tc_tables_t<16>(img);
    else tc_tables_t<32>(img);
}

template <int G, bool W, bool ZT = false>
static cudaError_t launch_cf_tc_t(const CFArgs &a, const void *tables, int *status, cudaStream_t s)
{
    using Shp = TcShape<G, W, ZT>;
    // 227 KB per CTA, less the kernel's 1 KB of static shared memory (barriers, aligned)
    static_assert(Shp::kSmem <= 232448 - 1024, "tensor-core filter: shared memory over the per-CTA limit");
    const size_t smem = (size_t)Shp::kSmem;
    cudaError_t e;
    if ((e = allow_smem(cf_tc_kernel<G, W, ZT>, smem)) != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    // one CTA per SM (shared memory and all 512 tensor-memory columns are taken)
    const long long ntiles = (a.ngroups + TcLayout<G>::kGroups - 1) / TcLayout<G>::kGroups;
    const long long grid = std::max<long long>(1, std::min<long long>((ntiles + Shp::kWG - 1) / Shp::kWG, sms));
    COUNT_LAUNCH();
    cf_tc_kernel<G, W, ZT><<<(unsigned)grid, Shp::kTeam * Shp::kWG, smem, s>>>(a, static_cast<const float4 *>(tables), ntiles, status);
    return cudaGetLastError();
}

int cf_tc_zt_supported(int B, int G, int wiener) { return B == 8 && G == 32 && wiener; }

cudaError_t launch_cf_tile_lists(const int *count, long long ngroups, int G, int *full, unsigned int *nfull,
                                 int *shrt, unsigned int *nshort, int *chunk_counts, cudaStream_t s)
{
    const long long ntiles = (ngroups + 128 / G - 1) / (128 / G);
    const long long chunks = std::max<long long>(1, (ntiles + kTileChunk - 1) / kTileChunk);
    COUNT_LAUNCH();
    cf_tile_count_kernel<<<(unsigned)chunks, 256, 0, s>>>(count, ngroups, G, ntiles, chunk_counts);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    COUNT_LAUNCH();
    cf_tile_lists_kernel<<<(unsigned)chunks, 256, 0, s>>>(count, ngroups, G, ntiles, chunk_counts, full, nfull, shrt, nshort);
    return cudaGetLastError();
}

long long cf_tile_chunks(long long ngroups, int G)
{
    const long long ntiles = (ngroups + 128 / G - 1) / (128 / G);
    return std::max<long long>(1, (ntiles + kTileChunk - 1) / kTileChunk);
}

cudaError_t launch_cf_tc_zt(const CFArgs &a, const void *tables, int *status, cudaStream_t s)
{
    if (!cf_tc_zt_supported(a.B, a.G, a.wiener)) return cudaErrorInvalidValue;
    return launch_cf_tc_t<32, true, true>(a, tables, status, s);
}

// Dz as [kz][b] and Ci as [b][kz], K-major without swizzle (the transposed z stage's B operands)
void cf_tc_zt_tables(int G, std::vector<float> &out)
{
    out.assign((size_t)2 * G * G, 0.0f);
    for (int r = 0; r < G; ++r)
        for (int k = 0; k < G; ++k) {
            out[tc_kmajor(r, k, G) / 4] = round_tf32((float)cos2((long)(2 * k + 1) * r, 2L * G));
            out[G * G + tc_kmajor(r, k, G) / 4] = round_tf32(k == 0 ? 1.0f : (float)cos2((long)k * (2 * r + 1), 2L * G));
        }
}

cudaError_t launch_cf_tc(const CFArgs &a, const void *tables, int *status, cudaStream_t s)
{
    if (!cf_tc_supported(a.B, a.G)) return cudaErrorInvalidValue;
    const bool w = a.wiener != 0;
    switch (a.G) {
    case 8: return w ? launch_cf_tc_t<8, true>(a, tables, status, s) : launch_cf_tc_t<8, false>(a, tables, status, s);
    case 16: return w ? launch_cf_tc_t<16, true>(a, tables, status, s) : launch_cf_tc_t<16, false>(a, tables, status, s);
    default: return w ? launch_cf_tc_t<32, true>(a, tables, status, s) : launch_cf_tc_t<32, false>(a, tables, status, s);
    }
}

// ---- FP64 oracle (inspection) --------------------------------------------------------------------

size_t cf_fp64_smem(int B, int G) { return sizeof(double) * ((size_t)2 * G * B * B + 64 * 64); }

cudaError_t launch_cf_fp64(const CFArgs &a, const F64Args &f, cudaStream_t s)
{
    const size_t smem = cf_fp64_smem(a.B, a.G);
    cudaError_t e;
    // always raised: the kernel's static shared memory comes on top of the dynamic part
    if ((e = cudaFuncSetAttribute(cf_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
        return e;
    COUNT_LAUNCH();
    cf_fp64_kernel<<<(unsigned)a.ngroups, 64, smem, s>>>(a, f);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    dim3 grid((a.W + 127) / 128, a.H, 3);
    COUNT_LAUNCH();
    finalize_fp64_kernel<<<grid, 128, 0, s>>>(f, a.W, a.H, 1, a.process[0], a.process[1], a.process[2]);
    return cudaGetLastError();
}

template <int BM, bool DIRECT>
static cudaError_t launch_cf_mid_t(const CFArgs &a, cudaStream_t s)
{
    auto kernel = a.wiener ? cf_mid_kernel<BM, DIRECT, true> : cf_mid_kernel<BM, DIRECT, false>;
    const size_t smem = mid_smem_bytes(BM, a.B, a.G, a.wiener);
    cudaError_t e;
    if ((e = allow_smem(kernel, smem)) != cudaSuccess) return e;
    COUNT_LAUNCH();
    kernel<<<(unsigned)std::max<long long>(1, std::min<long long>(a.ngroups, 148LL * 64)), kMidThreads, smem, s>>>(a);
    return cudaGetLastError();
}

int launch_cf_mid(const CFArgs &a, cudaStream_t s, cudaError_t *e)
{
    if (a.B < 2 || a.B > 16 || a.G > 32 || mid_smem_bytes(16, a.B, a.G, a.wiener) > 200 * 1024) return 0;
    switch (a.B) {
    case 2: *e = launch_cf_mid_t<2, false>(a, s); break;
    case 4: *e = launch_cf_mid_t<4, false>(a, s); break;
    case 8: *e = launch_cf_mid_t<8, false>(a, s); break;
    case 16: *e = launch_cf_mid_t<16, false>(a, s); break;
    default:
        *e = a.B < 4 ? launch_cf_mid_t<4, true>(a, s) : a.B < 8 ? launch_cf_mid_t<8, true>(a, s)
           : a.B <= 12 ? launch_cf_mid_t<12, true>(a, s) : launch_cf_mid_t<16, true>(a, s);
    }
    return 1;
}

cudaError_t launch_cf_generic(const CFArgs &a, int warps, int grid, cudaStream_t s)
{
    COUNT_LAUNCH();
    cf_generic_kernel<<<grid, 32 * warps, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_convert(const ConvProgram &pr, const PlanePtr *in, const PlanePtr *out, int nframes, cudaStream_t s)
{
    auto aligned = [](const PlanePtr &p, int kind) {
        const long long m = kind == SK_U8 ? 7 : 15;
        return !p.ptr || ((reinterpret_cast<long long>(p.ptr) | p.stride) & m) == 0;
    };
    const int per = kConvPlanes / std::max(pr.nin, pr.nout);
    const long long units = (long long)((pr.W + 7) >> 3) * pr.H;
    for (int f0 = 0; f0 < nframes; f0 += per) {
        const int nf = std::min(per, nframes - f0);
        ConvTable t{};
        bool vec = true;
        for (int k = 0; k < nf * pr.nin; ++k) {
            t.in[k] = in[f0 * pr.nin + k];
            vec = vec && aligned(t.in[k], pr.in_kind);
        }
        for (int k = 0; k < nf * pr.nout; ++k) {
            t.out[k] = out[f0 * pr.nout + k];
            vec = vec && aligned(t.out[k], pr.out_kind);
        }
        const dim3 grid((unsigned)((units + 255) / 256), nf);
        COUNT_LAUNCH();
        if (vec) convert_kernel<true><<<grid, 256, 0, s>>>(pr, t);
        else convert_kernel<false><<<grid, 256, 0, s>>>(pr, t);
    }
    return cudaGetLastError();
}

cudaError_t launch_finalize(const FinalizeArgs &a, int nframes, cudaStream_t s)
{
    const size_t smem = sizeof(float) * (size_t)finalize_smem_floats(a.B);
    cudaError_t e;
    if ((e = allow_smem(finalize_kernel, smem)) != cudaSuccess) return e;
    dim3 grid((a.W + kFinTW - 1) / kFinTW, (a.H + kFinTH - 1) / kFinTH, nframes * 3);
    COUNT_LAUNCH();
    finalize_kernel<<<grid, 256, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_vaggregate(const VAggArgs &a, int nframes, cudaStream_t s)
{
    dim3 block(256);
    dim3 grid((a.W + 255) / 256, a.H * 3, nframes);
    COUNT_LAUNCH();
    vaggregate_kernel<<<grid, block, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_vstack(const VStackArgs &a, int nframes, cudaStream_t s)
{
    const size_t smem = sizeof(float) * (size_t)finalize_smem_floats(a.B);
    cudaError_t e;
    if ((e = allow_smem(vstack_kernel, smem)) != cudaSuccess) return e;
    dim3 grid((a.W + kFinTW - 1) / kFinTW, a.slots * ((a.H + kFinTH - 1) / kFinTH), nframes * 3);
    COUNT_LAUNCH();
    vstack_kernel<<<grid, 256, smem, s>>>(a);
    return cudaGetLastError();
}

// ---- transform-only test kernels ------------------------------------------------------------

template <int G>
__global__ void dct_fast_test_kernel(float *data, int inverse)
{
    __shared__ float T[32 * 65];
    const int lane = threadIdx.x;
    float *g = data + (long long)blockIdx.x * G * 64;
    constexpr int C = 64 / G;
    if (!inverse) {
        if (lane < G) {
            float blk[64];
#pragma unroll
            for (int e = 0; e < 64; ++e) blk[e] = g[lane * 64 + e];
            fwd2d8(blk);
#pragma unroll
            for (int e = 0; e < 64; ++e) T[lane * 65 + e] = blk[e];
        }
        __syncwarp();
        if (lane < G) {
#pragma unroll
            for (int q = 0; q < C; ++q) {
                const int c = lane + q * G;
                float col[G], X[G];
#pragma unroll
                for (int zz = 0; zz < G; ++zz) col[zz] = T[zz * 65 + c];
                fdct_reg<G>(col, X);
#pragma unroll
                for (int zz = 0; zz < G; ++zz) g[zz * 64 + c] = X[zz];
            }
        }
    } else {
        if (lane < G) {
#pragma unroll
            for (int q = 0; q < C; ++q) {
                const int c = lane + q * G;
                float col[G], X[G];
#pragma unroll
                for (int zz = 0; zz < G; ++zz) X[zz] = g[zz * 64 + c];
                idct_reg<G>(X, col);
#pragma unroll
                for (int zz = 0; zz < G; ++zz) T[zz * 65 + c] = col[zz];
            }
        }
        __syncwarp();
        if (lane < G) {
            float blk[64];
#pragma unroll
            for (int e = 0; e < 64; ++e) blk[e] = T[lane * 65 + e];
            inv2d8(blk);
#pragma unroll
            for (int e = 0; e < 64; ++e) g[lane * 64 + e] = blk[e];
        }
    }
}

__global__ void dct_generic_test_kernel(float *data, int n, int B, int inverse, CFArgs a)
{
    float tmp[512];
    float *g = data + (long long)blockIdx.x * n * B * B;
    dct3d_warp(g, n, B, inverse != 0, a, tmp);
}

cudaError_t launch_dct3d_test(float *data, int ngroups, int n, int B, int inverse, int fast,
                              const float *odd_all, const float *dtab, const int *dtab_off,
                              cudaStream_t s)
{
    if (fast) {
        if (B != 8) return cudaErrorInvalidValue;
        switch (n) {
        case 8: dct_fast_test_kernel<8><<<ngroups, 32, 0, s>>>(data, inverse); break;
        case 16: dct_fast_test_kernel<16><<<ngroups, 32, 0, s>>>(data, inverse); break;
        case 32: dct_fast_test_kernel<32><<<ngroups, 32, 0, s>>>(data, inverse); break;
        default: return cudaErrorInvalidValue;
        }
    } else {
        CFArgs a{};
        a.odd_all = odd_all;
        a.dtab = dtab;
        a.dtab_off = dtab_off;
        dct_generic_test_kernel<<<ngroups, 32, 0, s>>>(data, n, B, inverse, a);
    }
    return cudaGetLastError();
}

// each pair as a column of one coefficient
__global__ void wiener_test_kernel(const float *r2, const float *sg, int n, float *w, float *exact)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float r[1] = {r2[i]};
    float v[1], q[1], top = wiener_top(sg[i]), unused = 0.0f;
    wiener_weights<false, 1>(r, sg[i], v, top);
    wiener_weights<true, 1>(r, sg[i], q, unused);
    w[i] = top < kWienerTop ? v[0] : q[0];
    exact[i] = q[0];
}

cudaError_t launch_wiener_test(const float *r2, const float *sg, int n, float *w, float *exact, cudaStream_t s)
{
    wiener_test_kernel<<<(n + 255) / 256, 256, 0, s>>>(r2, sg, n, w, exact);
    return cudaGetLastError();
}

}  // namespace bm3d
