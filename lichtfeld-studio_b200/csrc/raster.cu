// Alpha-blend rasterizer by ray / Gaussian distance: forward, backward and the per-Gaussian
// gradient epilogues.
//
// Replaces gsplat/RasterizeToPixelsFromWorld3DGSFwd.cu:20 (K7), gsplat/RasterizeToPixelsFromWorld3DGSBwd.cu:17
// (K8) with the VJPs of gsplat/Utils.cuh:104-194, gsplat/SphericalHarmonicsCUDA.cu:445 (K3) and the
// activation backward that autograd performs for src/core/splat_data.cpp:267-286.
//
// Design (bound by instruction issue and the shared-memory pipe; no tensor cores: the largest contraction is 3x3):
//  * a warp owns a patch of pixels and walks its tile's depth-sorted list by itself, 32 entries at a time: no barrier. (With the four or eight warps of a
//    tile on one staged batch, a seventh to a fifth of the warps' time was waiting for one another: 1 M Gaussians, 1296x840, backward 760 -> 721 us,
//    3 M at 1600x1064 2415 -> 1983, where warps also start at their own last contributor);
//  * the packed 64-byte records are built once per Gaussian, so no per-Gaussian work is repeated per tile or per pixel. A warp looks at the boxes of
//    32 entries and fetches the records of those that overlap its patch (EntryFeed); a ballot keeps the ones whose forms reach the cut on it
//    (patch_reached);
//  * per pair the response is exp(-|g|^2 phi / 2), phi = (e1^2 + e2^2) / (e1^2 + e2^2 + w^2) with three linear forms of the
//    pixel direction (RayFrame, gsmath.cuh): 10 instructions up to the exp-free rejection test for the planar camera models
//    against 23 for u = M d, u x g and the two norms;
//  * a thread owns one pixel or two horizontally adjacent ones, held in the halves of 64-bit registers and evaluated by the packed fp32 instructions
//    (launch_raster_fwd says where which). 1 M Gaussians, 1296x840: backward 719 us against 755 with two scalar evaluations, 579 M warp instructions
//    against 694; forward 352 against 388;
//  * backward: every (warp, Gaussian) contribution is 12 numbers that are LINEAR in the per-pixel terms (kSums). They
//    are summed over the warp by a transpose through padded shared-memory rows, in the shadow of the next entry's evaluation, and leave as one coalesced
//    reduction to the Gaussian's accumulator row. The nonlinear quaternion / scale VJP runs once per Gaussian in the epilogue instead of once
//    per pixel pair;
//  * a rolling shutter gives every pixel its own ray origin: its kernels (_rs) keep u = M d and 16 sums, one pixel per thread and the tile's list staged for
//    all warps.
#include "gsmath.cuh"
#include "raster.cuh"
#include "pixels.cuh"
#include <math_constants.h>

namespace lfs {

namespace {

constexpr int kBlock = 256;
constexpr float kAlphaMin = 1.f / 255.f;

__device__ __forceinline__ void pixel_of_thread(int tile, int tw, int& i, int& j) {
    // warps tile the 16x16 block as 2 x 4 patches of 8 x 4 pixels
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lx = (warp & 1) * 8 + (lane & 7);
    const int ly = (warp >> 1) * 4 + (lane >> 3);
    i = (tile / tw) * 16 + ly;
    j = (tile % tw) * 16 + lx;
}

// Warp patch of 8x4 pixels: inclusive pixel bounds packed like the Gaussian boxes (lo | hi << 16).
__device__ __forceinline__ void warp_patch(int tile, int tw, uint32_t& px, uint32_t& py) {
    const int warp = threadIdx.x >> 5;
    const uint32_t x0 = (tile % tw) * 16 + (warp & 1) * 8, y0 = (tile / tw) * 16 + (warp >> 1) * 4;
    px = x0 | ((x0 + 7) << 16);
    py = y0 | ((y0 + 3) << 16);
}
__device__ __forceinline__ bool box_overlaps(uint2 box, uint32_t px, uint32_t py) {
    return (box.x & 0xFFFFu) <= (px >> 16) && (box.x >> 16) >= (px & 0xFFFFu) &&
           (box.y & 0xFFFFu) <= (py >> 16) && (box.y >> 16) >= (py & 0xFFFFu);
}

// The three linear forms of a record (common.cuh) at a pixel direction. For the planar models d = (x, y, 1), p2.x = 0.
struct RayForms { float e1, e2, w, E, den; };
template <int MODEL>
__device__ __forceinline__ RayForms ray_forms(const float4& r0, const float4& r1, const float4& r2, const f3& d) {
    RayForms f;
    if (MODEL == LFS_PINHOLE || MODEL == LFS_PINHOLE_OPENCV) {
        f.e1 = r0.x * d.x + (r0.y * d.y + r0.z);
        f.e2 = r1.y * d.y + r1.z;
        f.w = r2.x * d.x + (r2.y * d.y + r2.z);
    } else {
        f.e1 = r0.x * d.x + (r0.y * d.y + r0.z * d.z);
        f.e2 = r1.x * d.x + (r1.y * d.y + r1.z * d.z);
        f.w = r2.x * d.x + (r2.y * d.y + r2.z * d.z);
    }
    f.E = f.e1 * f.e1 + f.e2 * f.e2;
    f.den = f.w * f.w + f.E;
    return f;
}

// The directions of a warp's patch as an axis-aligned box around a centre (camera space; depth 0 for the planar models), over
// the pixels that take part.
struct PatchRays { f3 c, h; };
__device__ __forceinline__ void patch_axis(float lo, float hi, float& c, float& h) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    c = 0.5f * (lo + hi);
    h = 0.5f * (hi - lo) * 1.00001f;
}
template <int MODEL, int PX>
__device__ __forceinline__ PatchRays patch_rays(const f3* d, const bool* takes_part) {
    f3 lo{1e30f, 1e30f, 1e30f}, hi{-1e30f, -1e30f, -1e30f};
#pragma unroll
    for (int p = 0; p < PX; ++p)
        if (takes_part[p]) {
            lo = f3{fminf(lo.x, d[p].x), fminf(lo.y, d[p].y), fminf(lo.z, d[p].z)};
            hi = f3{fmaxf(hi.x, d[p].x), fmaxf(hi.y, d[p].y), fmaxf(hi.z, d[p].z)};
        }
    PatchRays r;
    patch_axis(lo.x, hi.x, r.c.x, r.h.x);
    patch_axis(lo.y, hi.y, r.c.y, r.h.y);
    r.c.z = 1.f;
    r.h.z = 0.f;
    if (MODEL != LFS_PINHOLE && MODEL != LFS_PINHOLE_OPENCV) patch_axis(lo.z, hi.z, r.c.z, r.h.z);
    return r;
}
// Can a ray of the patch reach alpha >= 1/255? The forms are linear, so (e1, e2) of the patch lie in a parallelogram around its
// centre's e_c; along e_c it comes no closer to the origin than |e_c| - ext, and it is out of reach when that exceeds slope times
// the largest |w|. The axis-aligned screen box has already passed: this takes out its corners (slanted and round footprints).
// The rounding of the forms is covered by a multiple of their coefficients. Some 35 instructions per (entry, patch), one lane
// each, against the 40 - 140 of a walked entry: 1 M Gaussians at 1296x840 forward 429 -> 382 us, backward 816 -> 759; 6 M at 4K
// 1440 -> 1224; 6 M 180 degree fisheye, whose boxes are ring sectors, 1382 -> 1129.
template <int MODEL>
__device__ __forceinline__ bool patch_reached(const float4& r0, const float4& r1, const float4& r2, float slope, const PatchRays& P) {
    constexpr bool planar = MODEL == LFS_PINHOLE || MODEL == LFS_PINHOLE_OPENCV;
    const RayForms f = ray_forms<MODEL>(r0, r1, r2, P.c);
    const float inv = rsqrtf(fmaxf(f.E, 1e-37f));
    const float u1 = f.e1 * inv, u2 = f.e2 * inv;
    float ext = fabsf(u1 * r0.x + u2 * r1.x) * P.h.x + fabsf(u1 * r0.y + u2 * r1.y) * P.h.y;
    float w = fabsf(f.w) + fabsf(r2.x) * P.h.x + fabsf(r2.y) * P.h.y;
    if (!planar) { ext += fabsf(u1 * r0.z + u2 * r1.z) * P.h.z; w += fabsf(r2.z) * P.h.z; }
    const float slack = 1e-6f * (fabsf(r0.x) + fabsf(r0.y) + fabsf(r0.z) + fabsf(r1.x) + fabsf(r1.y) + fabsf(r1.z));
    return !(f.E * inv - ext > slope * w * 1.001f + slack);   // true for NaN
}

// Which side of alpha = 1/255 a pair near it falls on: |u x g|^2 / |u|^2 with u = M d in float32, d the pixel's world-space unit
// ray, as the kernels with one ray origin per pixel compute it. The three forms round differently (make_record bounds by how
// much), and a pair that changes side moves a pixel by up to 1/255 of a colour and the gradient of a small Gaussian by percents:
// the set of blended pairs must not depend on which expression is the faster one.
// The products and sums are spelled out, so that the set does not depend on a compiler's contraction either.
// For PX pixels of one thread, as bits. cut: the first row of the Gaussian's cut record, the others n apart; rays: stride apart.
// A call, since fewer than one walked entry in a hundred comes here and the registers of the callers' loops should not be shaped
// by it (1 M Gaussians, 1296x840, with the kernels of the time: backward 786 us against 845 inlined; forward 398 either way).
template <int PX>
__device__ __noinline__ uint32_t kept_at_cut(const float4* cut, int64_t n, const f3* rays, int stride, float opacity) {
    auto dot = [](float a0, float b0, float a1, float b1, float a2, float b2) { return fmaf(a2, b2, fmaf(a0, b0, __fmul_rn(a1, b1))); };
    auto det = [](float a, float b, float c, float e) { return fmaf(a, b, -__fmul_rn(c, e)); };
    const float4 r0 = cut[0], r1 = cut[n], r2 = cut[2 * n];
    uint32_t kept = 0;
#pragma unroll
    for (int p = 0; p < PX; ++p) {
        const f3 d = rays[p * stride];
        const float ux = dot(r0.x, d.x, r0.y, d.y, r0.z, d.z), uy = dot(r1.x, d.x, r1.y, d.y, r1.z, d.z), uz = dot(r2.x, d.x, r2.y, d.y, r2.z, d.z);
        const float cx = det(uy, r2.w, r1.w, uz), cy = det(uz, r0.w, r2.w, ux), cz = det(ux, r1.w, r0.w, uy);
        const float cc = dot(cx, cx, cy, cy, cz, cz), uu = dot(ux, ux, uy, uy, uz, uz);
        const float power = -0.5f * __fdividef(cc, fmaxf(uu, 1e-37f));
        if (!(fminf(0.999f, opacity * __expf(power)) < kAlphaMin)) kept |= 1u << p;
    }
    return kept;
}

__device__ __forceinline__ int32_t load_count(const int32_t* n_dev, int64_t n_host) {
    return n_dev ? *n_dev : (int32_t)n_host;
}

// ---------------------------------------------------------------------------------------------
// Staging of one batch of tile entries into shared memory with 16-byte asynchronous copies
// (cp.async: the entries are a gather by Gaussian index, so each copy is one quarter record or one
// bounds row). Two buffers: batch b+1 is in flight while batch b is being blended.
template <int BATCH>
struct Stage {
    float4 rec[BATCH * 4];  // packed records
    uint4 box[BATCH];       // rows of RasterArgs::bounds
};

// Each thread owns kParts quarter-record slots q = k * BLOCK + tid of a batch: entry q >> 2, part q & 3.
template <int BATCH, int BLOCK>
struct StageIds {
    static constexpr int kParts = (BATCH * 4 + BLOCK - 1) / BLOCK;
    uint32_t g[kParts];
};

// ids of the batch whose first list position is `first` and which runs forward (step +1) or backward (-1)
template <int BATCH, int BLOCK>
__device__ __forceinline__ void load_ids(StageIds<BATCH, BLOCK>& ids, const uint32_t* __restrict__ flatten_ids, int32_t first,
                                         int step, int batch_size) {
#pragma unroll
    for (int k = 0; k < StageIds<BATCH, BLOCK>::kParts; ++k) {
        const int e = (k * BLOCK + threadIdx.x) >> 2;
        ids.g[k] = e < batch_size ? flatten_ids[first + step * e] : 0u;
    }
}

template <int BATCH, int BLOCK>
__device__ __forceinline__ void issue_stage(Stage<BATCH>& st, uint32_t* sid, const StageIds<BATCH, BLOCK>& ids,
                                            const float4* __restrict__ records, const uint4* __restrict__ bounds,
                                            int batch_size) {
#pragma unroll
    for (int k = 0; k < StageIds<BATCH, BLOCK>::kParts; ++k) {
        const int q = k * BLOCK + threadIdx.x;
        const int e = q >> 2, part = q & 3;
        if (e < batch_size) {
            cp_async16(&st.rec[q], records + (size_t)ids.g[k] * 4 + part);
            if (part == 0) {
                cp_async16(&st.box[e], bounds + ids.g[k]);
                if (sid) sid[e] = ids.g[k];
            }
        }
    }
    cp_async_commit();
}

// ---------------------------------------------------------------------------------------------
template <int PX>
struct PixelForms { typename Pixels<PX>::V e1, e2, w, E, den; };
template <int MODEL, int PX>
__device__ __forceinline__ PixelForms<PX> pixel_forms(const float4& r0, const float4& r1, const float4& r2, typename Pixels<PX>::V dx,
                                                      typename Pixels<PX>::V dy, typename Pixels<PX>::V dz) {
    using P = Pixels<PX>;
    PixelForms<PX> f;
    if (MODEL == LFS_PINHOLE || MODEL == LFS_PINHOLE_OPENCV) {
        f.e1 = fma2(P::all(r0.x), dx, fma2(P::all(r0.y), dy, P::all(r0.z)));
        f.e2 = fma2(P::all(r1.y), dy, P::all(r1.z));
        f.w = fma2(P::all(r2.x), dx, fma2(P::all(r2.y), dy, P::all(r2.z)));
    } else {
        f.e1 = fma2(P::all(r0.x), dx, fma2(P::all(r0.y), dy, mul2(P::all(r0.z), dz)));
        f.e2 = fma2(P::all(r1.x), dx, fma2(P::all(r1.y), dy, mul2(P::all(r1.z), dz)));
        f.w = fma2(P::all(r2.x), dx, fma2(P::all(r2.y), dy, mul2(P::all(r2.z), dz)));
    }
    f.E = fma2(f.e1, f.e1, mul2(f.e2, f.e2));
    f.den = fma2(f.w, f.w, f.E);
    return f;
}

// A warp's own staging of 32 entries, part by part: lanes that read the same part of 32 entries (the culling) touch consecutive 16-byte
// words. With the four parts of an entry side by side those loads were 64 bytes apart and took four times as many passes.
struct WarpStage {
    float4 rec[4][32];
    float2 zw[32];       // slope and extra value of the entry's row of RasterArgs::bounds
    uint32_t sid[32];    // Gaussian
};
// Entries of a list for one warp, 32 at a time in three stages: the index of batch b + 3 and the box of b + 2 are on their way to registers and the records of
// b + 1 to shared memory while b is walked. Only entries whose box overlaps the patch are fetched.
struct EntryFeed {
    uint32_t id_box, id_ahead;   // of the batch whose boxes are on their way, and of the one after it
    uint4 box;
    uint32_t mask;               // entries of the batch staged last
    __device__ __forceinline__ void start(uint32_t id0, uint32_t id1, const uint4* __restrict__ bounds) {
        id_box = id0;
        id_ahead = id1;
        box = bounds[id0];
    }
    // stages the batch whose boxes have come (n entries), starts on the boxes of the next one; id: of the batch after that
    __device__ __forceinline__ void stage(WarpStage& st, int n, uint32_t patch_x, uint32_t patch_y, const float4* __restrict__ records,
                                          const uint4* __restrict__ bounds, uint32_t id, int lane) {
        const bool ov = lane < n && box_overlaps(make_uint2(box.x, box.y), patch_x, patch_y);
        mask = __ballot_sync(0xffffffffu, ov);
        if (ov) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cp_async16(&st.rec[k][lane], records + (size_t)id_box * 4 + k);
            st.zw[lane] = make_float2(__uint_as_float(box.z), __uint_as_float(box.w));
            st.sid[lane] = id_box;
        }
        cp_async_commit();
        id_box = id_ahead;
        id_ahead = id;
        box = bounds[id_box];
    }
};

template <int PX>
struct FwdPatchWarp {
    WarpStage stage[2];   // one is walked while the other is filled
    f3 ray[PX][32];       // world-space unit rays, for kept_at_cut
};

// Forward for cameras with one ray origin. A warp owns a patch of 8 x 4 PX pixels and stages its own entries: no barrier, and a warp whose pixels are finished
// stops by itself. EXTRA = false: three colour channels (render mode RGB). EXTRA = true: `channels` is 1 or 4 and the last
// channel blends the per-Gaussian value kept in bounds.w (the depth in the render modes D / ED / RGB_D /
// RGB_ED of gsplat/Rasterization.cpp:373-393); `normalize` divides it by max(alpha, 1e-10) on output (the
// expected-depth modes of src/training/rasterization/rasterizer.cpp:186-198) and keeps the undivided value
// in extra_sum for the backward.
// Pixels whose pair is rejected go on with alpha = 0. VOTE: the warp leaves an entry that reaches no pixel. A wide-angle camera's warps have many of those
// (6 M fisheye 1300 -> 1164 us), and so have the outsized lists (pixels.cuh), whose Gaussians are small beside a patch (two of 632 k entries 82 -> 55 ms); a planar
// camera's others have few (1 M, 1296x840: 352 us against 361 with the vote; 16 k at 256x256 52 against 56).
// Eight CTAs of 64 registers per SM; seven 378 us, nine the same. The other cameras' two-pixel kernels spill 16 to 36 bytes and still want eight: opencv
// 400 k 326 us against 340 with seven, 6 M fisheye 1143 against 1209.
template <int MODEL, bool EXTRA, int PX, bool VOTE>
__global__ void __launch_bounds__(128, 8) raster_fwd_patch_kernel(
    const CamDev* __restrict__ cams, const float4* __restrict__ records, const float4* __restrict__ cuts, int64_t n_cuts,
    const uint4* __restrict__ bounds, const uint32_t* __restrict__ flatten_ids,
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ n_isects_dev, int64_t n_isects_host,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const uint8_t* __restrict__ masks,
    const int32_t* __restrict__ tile_order, int channels, int normalize, int W, int H, int tw, int n_tiles, Outsized out,
    float* __restrict__ render, float* __restrict__ alphas, int32_t* __restrict__ last_ids, float* __restrict__ extra_sum) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using P = Pixels<PX>;
    using V = typename P::V;
    FwdPatchWarp<PX>& sm = reinterpret_cast<FwdPatchWarp<PX>*>(smem_raw)[threadIdx.x >> 5];

    side_by_side<PX>(out);
    if (overflow && *overflow) return;
    const int slot = PX == 2 ? blockIdx.x : blockIdx.x >> 1;
    const int tile = tile_order ? tile_order[slot] : slot;
    if (PX == 1 ? out.share > 0 : slot < out.slots) {
        const int32_t all = load_count(n_isects_dev, n_isects_host), n = (tile == n_tiles - 1 ? all : tile_offsets[tile + 1]) - tile_offsets[tile];
        if (is_outsized(n, all, out) != (PX == 1)) return;
    }
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) + (PX == 2 ? 0 : (blockIdx.x & 1) * 4);
    // warps tile the 16x16 block as patches of 8 x 4 PX pixels
    const int patch_x0 = (tile % tw) * 16 + (warp & 1) * 8, patch_y0 = (tile / tw) * 16 + (warp >> 1) * 4 * PX;
    const uint32_t patch_x = patch_x0 | ((patch_x0 + 7) << 16), patch_y = patch_y0 | ((patch_y0 + 4 * PX - 1) << 16);
    const int i = patch_y0 + (PX == 2 ? lane >> 2 : lane >> 3), j0 = patch_x0 + (PX == 2 ? 2 * (lane & 3) : lane & 7);
    if (masks && !masks[tile]) {
        // a tile labelled false shows the background (gsplat/RasterizeToPixelsFromWorld3DGSFwd.cu:147-155)
#pragma unroll
        for (int q = 0; q < PX; ++q)
            if (i < H && j0 + q < W) {
                const int pid = i * W + j0 + q;
                const int ch = EXTRA ? channels : 3;
                for (int k = 0; k < ch; ++k) render[pid * ch + k] = background ? background[k] : 0.f;
                alphas[pid] = 0.f;
                last_ids[pid] = 0;
                if (EXTRA && extra_sum) extra_sum[pid] = background ? background[ch - 1] : 0.f;
            }
        return;
    }
    const CamDev& cam = cams[0];
    f3 d[PX];
    bool takes_part[PX];
    float dc[3][PX];
    uint32_t cur_idx[PX];
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        f3 wd;
        takes_part[q] = pixel_cam_dir<MODEL>(cam, (float)(j0 + q) + 0.5f, (float)i + 0.5f, d[q], wd) && i < H && j0 + q < W;
        sm.ray[q][lane] = wd;
        dc[1][q] = d[q].y; dc[2][q] = d[q].z;
        // a pixel that takes no part, or no longer, has no direction: every comparison with its distance is false
        dc[0][q] = takes_part[q] ? d[q].x : CUDART_NAN_F;
        cur_idx[q] = 0;
    }
    const PatchRays rays = patch_rays<MODEL, PX>(d, takes_part);
    V dx = P::make(dc[0]);
    const V dy = P::make(dc[1]), dz = P::make(dc[2]), minus_one = P::all(-1.0f);
    V T = P::all(1.0f), pr = P::all(0.f), pg = P::all(0.f), pb = P::all(0.f), px = P::all(0.f);

    const int32_t n_isects = load_count(n_isects_dev, n_isects_host);
    const int32_t range_start = tile_offsets[tile];
    const int32_t range_end = (tile == n_tiles - 1) ? n_isects : tile_offsets[tile + 1];
    const int total = range_end - range_start, n_batches = (total + 31) / 32;
    auto batch_ids = [&](int b) { return lane < total - 32 * b ? flatten_ids[range_start + 32 * b + lane] : 0u; };
    EntryFeed feed;
    if (n_batches > 0) {
        feed.start(batch_ids(0), batch_ids(1), bounds);
        feed.stage(sm.stage[0], total, patch_x, patch_y, records, bounds, batch_ids(2), lane);
    }
    for (int b = 0; b < n_batches; ++b) {
        const int32_t batch_start = range_start + 32 * b;
        float left[PX];
        P::get(dx, left);
        bool any_left = false;
#pragma unroll
        for (int q = 0; q < PX; ++q) any_left = any_left || left[q] == left[q];
        if (!__any_sync(0xffffffffu, any_left)) break;
        const uint32_t staged = feed.mask;
        // everybody has read batch b - 1, whose buffer is filled next: a vote would not order memory
        __syncwarp();
        if (b + 1 < n_batches) {
            feed.stage(sm.stage[(b + 1) & 1], total - 32 * (b + 1), patch_x, patch_y, records, bounds, batch_ids(b + 3), lane);
            if (!staged) continue;
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        WarpStage& st = sm.stage[b & 1];
        // entries whose forms miss this warp's patch are dropped up front
        bool reached = staged >> lane & 1u;
        // an infinite or NaN colour (make_record marks it): zero times it is not zero, so it is added where a pair near the cut is decided
        if (reached && st.rec[2][lane].w == CUDART_INF_F) {
            st.rec[3][lane] = make_float4(0.f, 0.f, 0.f, st.rec[3][lane].w);
            st.zw[lane].y = 0.f;
        }
        if (reached) reached = patch_reached<MODEL>(st.rec[0][lane], st.rec[1][lane], st.rec[2][lane], st.zw[lane].x, rays);
        uint32_t bits = __ballot_sync(0xffffffffu, reached);
        __syncwarp();
        while (bits) {
            const int t = __ffs(bits) - 1;
            bits &= bits - 1;
            const float4 r0 = st.rec[0][t], r1 = st.rec[1][t], r2 = st.rec[2][t], r3 = st.rec[3][t];
            const PixelForms<PX> f = pixel_forms<MODEL, PX>(r0, r1, r2, dx, dy, dz);
            float E[PX], limit[PX], den[PX], ex[PX], vis[PX], alpha[PX];
            P::get(f.E, E);
            P::get(mul2(P::all(r1.w), f.den), limit);
            P::get(f.den, den);
            bool valid[PX], any_valid = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                valid[q] = E[q] <= limit[q];
                any_valid = any_valid || valid[q];
            }
            if (VOTE && !__any_sync(0xffffffffu, any_valid)) continue;
#pragma unroll
            for (int q = 0; q < PX; ++q) den[q] = rcp_approx(den[q]);
            P::get(mul2(P::all(r0.w), mul2(f.E, P::make(den))), ex);
#pragma unroll
            for (int q = 0; q < PX; ++q) vis[q] = exp2_approx(ex[q]);
            P::get(mul2(P::all(r3.w), P::make(vis)), alpha);
            bool near_cut = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                alpha[q] = fminf(0.999f, alpha[q]);
                near_cut = near_cut || (valid[q] && alpha[q] < r2.w);
            }
            if (near_cut) {
                const uint32_t kept = kept_at_cut<PX>(cuts + st.sid[t], n_cuts, &sm.ray[0][lane], 32, r3.w);
#pragma unroll
                for (int q = 0; q < PX; ++q) valid[q] = valid[q] && ((kept >> q & 1u) || !(alpha[q] < r2.w));
                if (r2.w == CUDART_INF_F) {
                    const float4 colour = records[(size_t)st.sid[t] * 4 + 3];
                    float tq[PX], c0[PX], c1[PX], c2[PX], c3[PX];
                    P::get(T, tq); P::get(pr, c0); P::get(pg, c1); P::get(pb, c2); P::get(px, c3);
#pragma unroll
                    for (int q = 0; q < PX; ++q) {
                        if (!valid[q] || tq[q] * (1.0f - alpha[q]) <= 1e-4f) continue;
                        const float w = tq[q] * alpha[q];
                        c0[q] += w * colour.x; c1[q] += w * colour.y; c2[q] += w * colour.z;
                        if (EXTRA) c3[q] += w * __uint_as_float(bounds[st.sid[t]].w);
                    }
                    pr = P::make(c0); pg = P::make(c1); pb = P::make(c2); px = P::make(c3);
                }
            }
#pragma unroll
            for (int q = 0; q < PX; ++q)
                if (!valid[q]) alpha[q] = 0.f;
            V al = P::make(alpha);
            V next_T = mul2(T, mul2(add2(al, minus_one), minus_one));
            float nt[PX];
            P::get(next_T, nt);
            bool stops = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) stops = stops || nt[q] <= 1e-4f;   // no pixel without alpha comes here: its T is above
            if (stops) {
                float x[PX], t0[PX];
                P::get(dx, x);
                P::get(T, t0);
#pragma unroll
                for (int q = 0; q < PX; ++q)
                    if (nt[q] <= 1e-4f) { valid[q] = false; alpha[q] = 0.f; nt[q] = t0[q]; x[q] = CUDART_NAN_F; }
                dx = P::make(x);
                al = P::make(alpha);
                next_T = P::make(nt);
            }
            const V w = mul2(al, T);
            pr = fma2(P::all(r3.x), w, pr); pg = fma2(P::all(r3.y), w, pg); pb = fma2(P::all(r3.z), w, pb);
            if (EXTRA) px = fma2(P::all(st.zw[t].y), w, px);
#pragma unroll
            for (int q = 0; q < PX; ++q) cur_idx[q] = valid[q] ? (uint32_t)(batch_start + t) : cur_idx[q];
            T = next_T;
        }
    }
    cp_async_wait<0>();
    float Tq[PX], rq[PX], gq[PX], bq[PX], xq[PX];
    P::get(T, Tq); P::get(pr, rq); P::get(pg, gq); P::get(pb, bq); P::get(px, xq);
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        if (!(i < H && j0 + q < W)) continue;
        const int pid = i * W + j0 + q;
        alphas[pid] = 1.0f - Tq[q];
        if (background && (!EXTRA || channels == 4)) { rq[q] += Tq[q] * background[0]; gq[q] += Tq[q] * background[1]; bq[q] += Tq[q] * background[2]; }
        if (!EXTRA) {
            render[pid * 3 + 0] = rq[q];
            render[pid * 3 + 1] = gq[q];
            render[pid * 3 + 2] = bq[q];
        } else {
            if (channels == 4) {
                render[pid * 4 + 0] = rq[q];
                render[pid * 4 + 1] = gq[q];
                render[pid * 4 + 2] = bq[q];
            }
            if (background) xq[q] += Tq[q] * background[channels - 1];
            if (extra_sum) extra_sum[pid] = xq[q];
            render[pid * channels + channels - 1] = normalize ? xq[q] / fmaxf(1.0f - Tq[q], 1e-10f) : xq[q];
        }
        last_ids[pid] = (int32_t)cur_idx[q];
    }
}

// ---------------------------------------------------------------------------------------------
// EXTRA = false: three colour channels (render mode RGB). EXTRA = true: `channels` is 1 or 4 and the last
// channel blends the per-Gaussian value kept in bounds.w (the depth in the render modes D / ED / RGB_D /
// RGB_ED of gsplat/Rasterization.cpp:373-393); `normalize` divides it by max(alpha, 1e-10) on output (the
// expected-depth modes of src/training/rasterization/rasterizer.cpp:186-198) and keeps the undivided value
// in extra_sum for the backward.
// A rolling shutter: every pixel has its own pose, hence its own ray origin; the record's gro = M (o_start - mu) is
// corrected per pair by M (o_pixel - o_start).
template <int MODEL, bool EXTRA>
__global__ void __launch_bounds__(kBlock, 4) raster_fwd_rs_kernel(
    const CamDev* __restrict__ cams, const float4* __restrict__ records, const uint4* __restrict__ bounds, const uint32_t* __restrict__ flatten_ids,
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ n_isects_dev, int64_t n_isects_host,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const uint8_t* __restrict__ masks,
    const int32_t* __restrict__ tile_order, int channels, int normalize, int W, int H, int tw, int n_tiles,
    float* __restrict__ render, float* __restrict__ alphas, int32_t* __restrict__ last_ids, float* __restrict__ extra_sum) {
    constexpr int BATCH = 192;
    __shared__ Stage<BATCH> stage[2];

    if (overflow && *overflow) return;
    const int tile = tile_order ? tile_order[blockIdx.x] : blockIdx.x;
    int i, j;
    pixel_of_thread(tile, tw, i, j);
    const bool inside = (i < H && j < W);
    if (masks && !masks[tile]) {
        // a tile labelled false shows the background (gsplat/RasterizeToPixelsFromWorld3DGSFwd.cu:147-155)
        if (inside) {
            const int pid = i * W + j;
            const int ch = EXTRA ? channels : 3;
            for (int k = 0; k < ch; ++k) render[pid * ch + k] = background ? background[k] : 0.f;
            alphas[pid] = 0.f;
            last_ids[pid] = 0;
            if (EXTRA && extra_sum) extra_sum[pid] = background ? background[ch - 1] : 0.f;
        }
        return;
    }
    const CamDev& cam = cams[0];
    f3 d, oo{0.f, 0.f, 0.f};
    const bool ray_ok = pixel_world_ray_rs<MODEL>(cam, (float)j + 0.5f, (float)i + 0.5f, d, oo);
    bool done = !inside || !ray_ok;
    uint32_t patch_x, patch_y;
    warp_patch(tile, tw, patch_x, patch_y);

    const int32_t n_isects = load_count(n_isects_dev, n_isects_host);
    const int32_t range_start = tile_offsets[tile];
    const int32_t range_end = (tile == n_tiles - 1) ? n_isects : tile_offsets[tile + 1];
    const int n_batches = (range_end - range_start + BATCH - 1) / BATCH;

    float T = 1.0f;
    uint32_t cur_idx = 0;
    float pr = 0.f, pg = 0.f, pb = 0.f, px = 0.f;

    StageIds<BATCH, kBlock> ids;
    if (n_batches > 0) {
        load_ids(ids, flatten_ids, range_start, 1, min(BATCH, range_end - range_start));
        issue_stage(stage[0], nullptr, ids, records, bounds, min(BATCH, range_end - range_start));
        if (n_batches > 1) load_ids(ids, flatten_ids, range_start + BATCH, 1, min(BATCH, range_end - range_start - BATCH));
    }
    for (int b = 0; b < n_batches; ++b) {
        const int32_t batch_start = range_start + b * BATCH;
        const int32_t batch_size = min(BATCH, range_end - batch_start);
        // next batch into the other buffer (its previous contents were consumed before the barrier that ended
        // the previous iteration), then the ids of the batch after that
        if (b + 1 < n_batches) {
            issue_stage(stage[(b + 1) & 1], nullptr, ids, records, bounds, min(BATCH, range_end - batch_start - BATCH));
            if (b + 2 < n_batches)
                load_ids(ids, flatten_ids, batch_start + 2 * BATCH, 1, min(BATCH, range_end - batch_start - 2 * BATCH));
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        // everyone's copies of batch b have landed; leave early when every pixel of the tile is finished
        if (__syncthreads_count(done) >= kBlock) break;
        const Stage<BATCH>& st = stage[b & 1];
        if (!__all_sync(0xffffffffu, done)) {
            // entries of this batch whose box overlaps this warp's 8x4 patch: one ballot word per 32 entries, formed when its
            // turn comes (six words kept at once are five registers more, at 40 in all: 413 us against 398)
            auto reach = [&](int w) {
                const int e = w * 32 + (threadIdx.x & 31);
                bool ov = false;
                if (e < batch_size) {
                    const uint4 bx = st.box[e];
                    ov = box_overlaps(make_uint2(bx.x, bx.y), patch_x, patch_y);
                }
                return __ballot_sync(0xffffffffu, ov);
            };
#pragma unroll
            for (int w = 0; w < BATCH / 32; ++w) {
                uint32_t bits = reach(w);
                while (bits && !done) {
                    const int t = w * 32 + __ffs(bits) - 1;
                    bits &= bits - 1;
                    const float4 r0 = st.rec[t * 4 + 0], r1 = st.rec[t * 4 + 1], r2 = st.rec[t * 4 + 2];
                    const float ux = r0.x * d.x + r0.y * d.y + r0.z * d.z;
                    const float uy = r1.x * d.x + r1.y * d.y + r1.z * d.z;
                    const float uz = r2.x * d.x + r2.y * d.y + r2.z * d.z;
                    const float gx = r0.w + (r0.x * oo.x + r0.y * oo.y + r0.z * oo.z);
                    const float gy = r1.w + (r1.x * oo.x + r1.y * oo.y + r1.z * oo.z);
                    const float gz = r2.w + (r2.x * oo.x + r2.y * oo.y + r2.z * oo.z);
                    const float cx = uy * gz - gy * uz;
                    const float cy = uz * gx - gz * ux;
                    const float cz = ux * gy - gx * uy;
                    const float cc = cx * cx + cy * cy + cz * cz;
                    const float uu = ux * ux + uy * uy + uz * uz;
                    // power = -0.5 cc / uu ; reject when power < thr  <=>  cc > -2 thr uu
                    if (cc > -2.0f * __uint_as_float(st.box[t].z) * uu) continue;
                    const float power = -0.5f * __fdividef(cc, fmaxf(uu, 1e-37f));
                    const float alpha = fminf(0.999f, st.rec[t * 4 + 3].w * __expf(power));
                    if (alpha < kAlphaMin) continue;
                    const float4 r3 = st.rec[t * 4 + 3];
                    const float next_T = T * (1.0f - alpha);
                    if (next_T <= 1e-4f) { done = true; break; }
                    const float vis = alpha * T;
                    pr += r3.x * vis; pg += r3.y * vis; pb += r3.z * vis;
                    if (EXTRA) px += __uint_as_float(st.box[t].w) * vis;
                    cur_idx = (uint32_t)(batch_start + t);
                    T = next_T;
                }
            }
        }
        __syncthreads();  // buffer b & 1 may be refilled by the next iteration's issue
    }
    cp_async_wait<0>();
    if (inside) {
        const int pid = i * W + j;
        alphas[pid] = 1.0f - T;
        if (!EXTRA) {
            if (background) { pr += T * background[0]; pg += T * background[1]; pb += T * background[2]; }
            render[pid * 3 + 0] = pr;
            render[pid * 3 + 1] = pg;
            render[pid * 3 + 2] = pb;
        } else {
            if (channels == 4) {
                if (background) { pr += T * background[0]; pg += T * background[1]; pb += T * background[2]; }
                render[pid * 4 + 0] = pr;
                render[pid * 4 + 1] = pg;
                render[pid * 4 + 2] = pb;
            }
            if (background) px += T * background[channels - 1];
            if (extra_sum) extra_sum[pid] = px;
            render[pid * channels + channels - 1] = normalize ? px / fmaxf(1.0f - T, 1e-10f) : px;
        }
        last_ids[pid] = (int32_t)cur_idx;
    }
}

// ---------------------------------------------------------------------------------------------
// NS values per lane -> per-value sums over the warp, value k left in lanes 2k and 2k+1 (lanes from 2 NS on repeat the last).
// The transpose goes through shared memory owned by the warp instead of a shuffle butterfly (for 16 values about 40 issue
// slots against 90): row k (36 floats, 32 used) holds value k of the 32 lanes. The row stride of 36 floats puts the 16-byte
// loads of one quarter-warp (lane = 2 k + h reads the 16 lanes of half h of row k) on eight different bank groups, and
// the scalar stores of one row are contiguous. The closing shuffle needs every lane's sum, hence every lane's loads,
// before any lane returns, so the next call may overwrite the rows.
constexpr int kRedStride = 36;
template <int NS>
__device__ __forceinline__ float warp_reduce(const float (&v)[NS], float* __restrict__ red, int lane) {
#pragma unroll
    for (int k = 0; k < NS; ++k) red[k * kRedStride + lane] = v[k];
    __syncwarp();
    const float4* half = reinterpret_cast<const float4*>(red + min(lane >> 1, NS - 1) * kRedStride + 16 * (lane & 1));
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 x = half[q];
        s += (x.x + x.y) + (x.z + x.w);
    }
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

__device__ __forceinline__ float __reduce_add_sync_f32(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Sums per (warp, Gaussian). One ray origin: 12 = sums over the pixels of, with q = vis dL/dalpha (the opacity term),
// omega = w / den and phi = E / den,
//   q omega e1, q omega e2 | the same two times phi | q omega^2 e1^2, q omega^2 e1 e2, q omega^2 e2^2 | q phi | rgb | q
// Rolling shutter: 16 = sum v_u (x) d, sum v_gro, rgb, opacity.
constexpr int kSums = 12, kSumsRs = 16;
template <int BATCH>
struct BwdShared {
    Stage<BATCH> stage[3];       // batch b is walked while b+1 and b+2 are in flight
    uint32_t sid[3][BATCH];      // Gaussian index per slot
    float red[kBlock / 32][kSumsRs * kRedStride];  // per-warp transpose rows of warp_reduce
};

// 1 / x for x in [0.001, 1]: the hardware estimate and one Newton step (relative error below 2^-23).
__device__ __forceinline__ float rcp_newton(float x) {
    const float y = rcp_approx(x);
    return fmaf(y, fmaf(-x, y, 1.0f), y);
}

// Backward under a rolling shutter. EXTRA: the output has 1 or 4 channels and its last one blends bounds.w (see the forward). XGRAD: also return
// the gradient of that per-Gaussian value in accum_extra [N] (operator-level colours with 1 or 4 channels;
// the fused render modes drop it like gsplat/Rasterization.cpp:575-590 does).
template <int MODEL, int BATCH, bool EXTRA, bool XGRAD>
__global__ void __launch_bounds__(kBlock) raster_bwd_rs_kernel(
    const CamDev* __restrict__ cams, const float4* __restrict__ records, const uint4* __restrict__ bounds, const uint32_t* __restrict__ flatten_ids,
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ n_isects_dev, int64_t n_isects_host,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const uint8_t* __restrict__ masks,
    const int32_t* __restrict__ tile_order, int channels, int normalize, int W, int H, int tw, int n_tiles,
    const float* __restrict__ render_alphas, const int32_t* __restrict__ last_ids, const float* __restrict__ extra_sum,
    const float* __restrict__ v_render, const float* __restrict__ v_alphas, float* __restrict__ accum,
    float* __restrict__ accum_extra) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Shared = BwdShared<BATCH>;
    Shared& sm = *reinterpret_cast<Shared*>(smem_raw);

    if (overflow && *overflow) return;
    const int tile = tile_order ? tile_order[blockIdx.x] : blockIdx.x;
    if (masks && !masks[tile]) return;  // gsplat/RasterizeToPixelsFromWorld3DGSBwd.cu:84
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // warps tile the 16x16 block as patches of 4 x 8 pixels
    const int patch_x0 = (tile % tw) * 16 + (warp & 3) * 4, patch_y0 = (tile / tw) * 16 + (warp >> 2) * 8;
    const uint32_t patch_x = patch_x0 | ((patch_x0 + 3) << 16), patch_y = patch_y0 | ((patch_y0 + 7) << 16);
    const int i = patch_y0 + (lane >> 2), j = patch_x0 + (lane & 3);
    const CamDev& cam = cams[0];

    f3 d, oo;
    const bool ray_ok = pixel_world_ray_rs<MODEL>(cam, (float)j + 0.5f, (float)i + 0.5f, d, oo);
    const bool active = i < H && j < W && ray_ok;
    // What a lens leaves for a pixel without a ray may be anything, NaN too. Such a pixel's terms are multiplied by zero below,
    // which takes finite ones.
    if (!active) { d = f3{0.f, 0.f, 1.f}; oo = f3{0.f, 0.f, 0.f}; }
    const int pid = min(i * W + j, W * H - 1);
    const float T_final = 1.0f - render_alphas[pid];
    float T = T_final, vcr = 0.f, vcg = 0.f, vcb = 0.f, vcx = 0.f;
    const int32_t bin_final = active ? last_ids[pid] : -1;   // last list position that reached the pixel; below every position for pixels that take no part
    float v_a = v_alphas ? v_alphas[pid] : 0.f;
    if (!EXTRA) {
        vcr = v_render[pid * 3 + 0]; vcg = v_render[pid * 3 + 1]; vcb = v_render[pid * 3 + 2];
    } else {
        if (channels == 4) { vcr = v_render[pid * 4 + 0]; vcg = v_render[pid * 4 + 1]; vcb = v_render[pid * 4 + 2]; }
        vcx = v_render[pid * channels + channels - 1];
        if (normalize) {
            // output = sum / max(alpha, 1e-10): chain rule of the division and of clamp_min
            const float a = 1.0f - T_final, ac = fmaxf(a, 1e-10f);
            if (a > 1e-10f) v_a -= extra_sum[pid] / (ac * ac) * vcx;
            vcx = vcx / ac;
        }
    }
    float bg_dot = 0.f;
    if (background) {
        if (!EXTRA || channels == 4) bg_dot = background[0] * vcr + background[1] * vcg + background[2] * vcb;
        if (EXTRA) bg_dot += background[channels - 1] * vcx;
    }
    // what lies behind the entry being walked, as seen by the output gradient: T_final (v_a - background . v_colour), minus
    // (colour . v_colour) alpha T of every entry behind
    float behind = T_final * (v_a - bg_dot);
    const int32_t warp_bin_final = __reduce_max_sync(0xffffffffu, max(bin_final, 0));

    const int32_t n_isects = load_count(n_isects_dev, n_isects_host);
    const int32_t range_start = tile_offsets[tile];
    const int32_t range_end = (tile == n_tiles - 1) ? n_isects : tile_offsets[tile + 1];
    const int n_batches = (range_end - range_start + BATCH - 1) / BATCH;
    float* red = sm.red[warp];

    // batches run back to front: slot e of batch b holds list position batch_end - e
    StageIds<BATCH, kBlock> ids;
    auto batch_count = [&](int k) { return min(BATCH, range_end - k * BATCH - range_start); };
    auto batch_top = [&](int k) { return range_end - 1 - k * BATCH; };
    if (n_batches > 0) {
        load_ids(ids, flatten_ids, batch_top(0), -1, batch_count(0));
        issue_stage(sm.stage[0], sm.sid[0], ids, records, bounds, batch_count(0));
        if (n_batches > 1) {
            load_ids(ids, flatten_ids, batch_top(1), -1, batch_count(1));
            issue_stage(sm.stage[1], sm.sid[1], ids, records, bounds, batch_count(1));
            if (n_batches > 2) load_ids(ids, flatten_ids, batch_top(2), -1, batch_count(2));
        }
    }
    // One barrier per batch: after it, batch b is in shared memory and every warp has finished walking batch b-1,
    // so batch b+2 may be staged over b-1's records.
    for (int b = 0; b < n_batches; ++b) {
        const int32_t batch_end = batch_top(b);
        const int32_t batch_size = batch_count(b);
        if (b + 1 < n_batches) cp_async_wait<1>(); else cp_async_wait<0>();
        __syncthreads();
        if (b + 2 < n_batches) {
            issue_stage(sm.stage[(b + 2) % 3], sm.sid[(b + 2) % 3], ids, records, bounds, batch_count(b + 2));
            if (b + 3 < n_batches) load_ids(ids, flatten_ids, batch_top(b + 3), -1, batch_count(b + 3));
        }
        const Stage<BATCH>& st = sm.stage[b % 3];
        const uint32_t* sid = sm.sid[b % 3];
        // entries (back to front) that no pixel of this warp reaches (beyond its last contributor) or whose
        // box misses this warp's patch are dropped up front: one ballot word per 32 entries
        const int t_begin = max(0, batch_end - warp_bin_final);
        uint32_t live[BATCH / 32];
#pragma unroll
        for (int w = 0; w < BATCH / 32; ++w) {
            const int e = w * 32 + lane;
            bool ov = false;
            if (e >= t_begin && e < batch_size) {
                const uint4 bx = st.box[e];
                ov = box_overlaps(make_uint2(bx.x, bx.y), patch_x, patch_y);
            }
            live[w] = __ballot_sync(0xffffffffu, ov);
        }
#pragma unroll
        for (int w = 0; w < BATCH / 32; ++w) {
            uint32_t bits = live[w];
            while (bits) {
                const int t = w * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                // Every lane evaluates the pair (the record reads are warp-wide broadcasts); pixels that are outside
                // the image, beyond their last contributor or below the alpha threshold continue with alpha = vis = 0,
                // which makes every term they add exactly zero, so no per-lane branching is needed below.
                const float4 r0 = st.rec[t * 4 + 0], r1 = st.rec[t * 4 + 1], r2 = st.rec[t * 4 + 2];
                const float ux = r0.x * d.x + r0.y * d.y + r0.z * d.z;
                const float uy = r1.x * d.x + r1.y * d.y + r1.z * d.z;
                const float uz = r2.x * d.x + r2.y * d.y + r2.z * d.z;
                const float gx = r0.w + (r0.x * oo.x + r0.y * oo.y + r0.z * oo.z);
                const float gy = r1.w + (r1.x * oo.x + r1.y * oo.y + r1.z * oo.z);
                const float gz = r2.w + (r2.x * oo.x + r2.y * oo.y + r2.z * oo.z);
                const float cx = uy * gz - gy * uz;
                const float cy = uz * gx - gz * ux;
                const float cz = ux * gy - gx * uy;
                const float cc = cx * cx + cy * cy + cz * cz;
                const float uu = ux * ux + uy * uy + uz * uz;
                bool valid = (batch_end - t <= bin_final) && !(cc > -2.0f * __uint_as_float(st.box[t].z) * uu);
                if (!__any_sync(0xffffffffu, valid)) continue;
                const float inv = rsqrtf(fmaxf(uu, 1e-37f));
                const float4 r3 = st.rec[t * 4 + 3];
                float vis = __expf(-0.5f * (cc * (inv * inv)));
                float alpha = fminf(0.999f, r3.w * vis);
                valid = valid && !(alpha < kAlphaMin);
                if (!__any_sync(0xffffffffu, valid)) continue;
                if (!valid) { vis = 0.f; alpha = 0.f; }
                const float ra = rcp_newton(1.0f - alpha);
                T *= ra;
                const float fac = alpha * T;
                // colour . v_colour of this entry: the colours only ever meet the output gradient in this product
                float cv = r3.x * vcr + r3.y * vcg + r3.z * vcb;
                if (EXTRA) cv += __uint_as_float(st.box[t].w) * vcx;
                const float v_alpha = cv * T + ra * behind;
                behind -= cv * fac;
                // geometry and opacity only while alpha is not clamped at 0.999
                const float gate = (r3.w * vis <= 0.999f) ? vis : 0.f;
                const float q = gate * v_alpha;
                const float s = -(r3.w * q);  // v_c = s * c with c = n x g
                // with n = u / |u|, gn = g . n and w = gn n - g (minus the part of g orthogonal to n):
                //   v_g = v_c x n = -s w,   v_u = (v_n - (v_n . n) n) / |u| = (s gn / |u|) w
                const float nx = ux * inv, ny = uy * inv, nz = uz * inv;
                const float gn = gx * nx + gy * ny + gz * nz;
                const float wx = gn * nx - gx, wy = gn * ny - gy, wz = gn * nz - gz;
                const float ku = s * gn * inv;
                const float vu[3] = {ku * wx, ku * wy, ku * wz}, vg[3] = {-s * wx, -s * wy, -s * wz};
                const float dd[3] = {d.x, d.y, d.z}, od[3] = {oo.x, oo.y, oo.z};
                float v[kSumsRs];
                // g = M (o_start - mu) + M (o_pixel - o_start): the second term adds v_g (x) (o_pixel - o_start) to v_M
#pragma unroll
                for (int r = 0; r < 3; ++r) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[r * 3 + c] = vu[r] * dd[c] + vg[r] * od[c];
                    v[9 + r] = vg[r];
                }
                v[12] = fac * vcr; v[13] = fac * vcg; v[14] = fac * vcb; v[15] = q;
                const uint32_t g = sid[t];
                if (XGRAD) {
                    const float xs = __reduce_add_sync_f32(fac * vcx);
                    if (lane == 0) atomicAdd(accum_extra + g, xs);
                }
                const float total = warp_reduce<kSumsRs>(v, red, lane);
                if ((lane & 1) == 0) atomicAdd(accum + (size_t)g * 16 + (lane >> 1), total);
            }
        }
    }
    cp_async_wait<0>();
}

template <int PX>
struct BwdPatchWarp {
    WarpStage stage[2];                      // one is walked while the other is filled
    float red[kSums * kRedStride];           // transpose rows
    f3 ray[PX][32];                            // world-space unit rays, for kept_at_cut
};

// Backward for cameras with one ray origin. A warp owns a patch of 4 PX x 8 pixels. Each warp stages its own entries, from its own last contributor on: no
// barrier, the warps of a tile run apart. EXTRA, XGRAD: as below (raster_bwd_rs_kernel).
// Five CTAs of 96 registers per SM (PX = 2: 1 M Gaussians 719 us, six of 80 737, four 751).
// Predicating the eight idle lanes off the loads of `flush` saves a tenth of the shared-memory passes and loses more to the order it imposes (741).
template <int MODEL, bool EXTRA, bool XGRAD, int PX>
__global__ void __launch_bounds__(128, PX == 2 ? 5 : 6) raster_bwd_patch_kernel(
    const CamDev* __restrict__ cams, const float4* __restrict__ records, const float4* __restrict__ cuts, int64_t n_cuts,
    const uint4* __restrict__ bounds, const uint32_t* __restrict__ flatten_ids,
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ n_isects_dev, int64_t n_isects_host,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const uint8_t* __restrict__ masks,
    const int32_t* __restrict__ tile_order, int channels, int normalize, int W, int H, int tw, int n_tiles, Outsized out,
    const float* __restrict__ render_alphas, const int32_t* __restrict__ last_ids, const float* __restrict__ extra_sum,
    const float* __restrict__ v_render, const float* __restrict__ v_alphas, float* __restrict__ accum,
    float* __restrict__ accum_extra) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using P = Pixels<PX>;
    using V = typename P::V;
    BwdPatchWarp<PX>& sm = reinterpret_cast<BwdPatchWarp<PX>*>(smem_raw)[threadIdx.x >> 5];

    side_by_side<PX>(out);
    if (overflow && *overflow) return;
    const int slot = PX == 2 ? blockIdx.x : blockIdx.x >> 1;
    const int tile = tile_order ? tile_order[slot] : slot;
    const int32_t n_isects = load_count(n_isects_dev, n_isects_host);
    const int32_t range_start = tile_offsets[tile];
    const int32_t range_end = (tile == n_tiles - 1) ? n_isects : tile_offsets[tile + 1];
    if ((PX == 1 ? out.share > 0 : slot < out.slots) && is_outsized(range_end - range_start, n_isects, out) != (PX == 1)) return;
    if (masks && !masks[tile]) return;  // gsplat/RasterizeToPixelsFromWorld3DGSBwd.cu:84
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) + (PX == 2 ? 0 : (blockIdx.x & 1) * 4);
    const CamDev& cam = cams[0];

    // warps tile the 16x16 block as patches of 4 PX x 8 pixels
    constexpr int kPatchesX = 4 / PX;
    const int patch_x0 = (tile % tw) * 16 + (warp % kPatchesX) * 4 * PX, patch_y0 = (tile / tw) * 16 + (warp / kPatchesX) * 8;
    const uint32_t patch_x = patch_x0 | ((patch_x0 + 4 * PX - 1) << 16), patch_y = patch_y0 | ((patch_y0 + 7) << 16);
    const int i = patch_y0 + (lane >> 2), j0 = patch_x0 + PX * (lane & 3);
    f3 d[PX];
    bool takes_part[PX];
    float Tf[PX], vr[PX], vg[PX], vb[PX], vx[PX], bh[PX], dc[3][PX];
    int32_t bin_final[PX];   // last list position that reached the pixel; below every position for pixels that take no part
    int32_t warp_bin_final = -1;
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        const int j = j0 + q;
        f3 wd;
        const bool active = pixel_cam_dir<MODEL>(cam, (float)j + 0.5f, (float)i + 0.5f, d[q], wd) && i < H && j < W;
        sm.ray[q][lane] = wd;
        takes_part[q] = active;
        // What a lens leaves for a pixel without a ray may be anything, NaN too. Such a pixel's terms are multiplied by zero below,
        // which takes finite ones.
        if (!active) d[q] = f3{0.f, 0.f, 1.f};
        const int pid = min(i * W + j, W * H - 1);
        Tf[q] = 1.0f - render_alphas[pid];
        bin_final[q] = active ? last_ids[pid] : -1;
        warp_bin_final = max(warp_bin_final, bin_final[q]);
        float v_a = v_alphas ? v_alphas[pid] : 0.f;
        vx[q] = 0.f;
        if (!EXTRA) {
            vr[q] = v_render[pid * 3 + 0]; vg[q] = v_render[pid * 3 + 1]; vb[q] = v_render[pid * 3 + 2];
        } else {
            vr[q] = vg[q] = vb[q] = 0.f;
            if (channels == 4) { vr[q] = v_render[pid * 4 + 0]; vg[q] = v_render[pid * 4 + 1]; vb[q] = v_render[pid * 4 + 2]; }
            vx[q] = v_render[pid * channels + channels - 1];
            if (normalize) {
                // output = sum / max(alpha, 1e-10): chain rule of the division and of clamp_min
                const float a = 1.0f - Tf[q], ac = fmaxf(a, 1e-10f);
                if (a > 1e-10f) v_a -= extra_sum[pid] / (ac * ac) * vx[q];
                vx[q] = vx[q] / ac;
            }
        }
        float bg_dot = 0.f;
        if (background) {
            if (!EXTRA || channels == 4) bg_dot = background[0] * vr[q] + background[1] * vg[q] + background[2] * vb[q];
            if (EXTRA) bg_dot += background[channels - 1] * vx[q];
        }
        bh[q] = Tf[q] * (v_a - bg_dot);
        dc[0][q] = d[q].x; dc[1][q] = d[q].y; dc[2][q] = d[q].z;
        vr[q] = -vr[q]; vg[q] = -vg[q]; vb[q] = -vb[q]; vx[q] = -vx[q];
    }
    const V dx = P::make(dc[0]), dy = P::make(dc[1]), dz = P::make(dc[2]);
    const V vcr = P::make(vr), vcg = P::make(vg), vcb = P::make(vb), vcx = P::make(vx);   // with the sign turned
    V T = P::make(Tf);
    // what lies behind the entry being walked, as seen by the output gradient: T_final (v_a - background . v_colour), minus
    // (colour . v_colour) alpha T of every entry behind
    V behind = P::make(bh);
    warp_bin_final = __reduce_max_sync(0xffffffffu, warp_bin_final);
    const PatchRays rays = patch_rays<MODEL, PX>(d, takes_part);

    // back to front from the patch's last contributor: slot e of batch b holds list position top - 32 b - e
    const int32_t top = min(range_end - 1, warp_bin_final);
    const int total = top - range_start + 1, n_batches = (total + 31) / 32;
    if (total <= 0) return;
    auto batch_ids = [&](int b) { return lane < total - 32 * b ? flatten_ids[top - 32 * b - lane] : 0u; };

    const V one = P::all(1.0f), minus_one = P::all(-1.0f);
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t pending = kNone;   // Gaussian whose sums lie in `red`
    const ulonglong2* red_half = reinterpret_cast<const ulonglong2*>(sm.red + min(lane >> 1, kSums - 1) * kRedStride + 16 * (lane & 1));
    const bool red_lane = (lane & 1) == 0 && lane < 2 * kSums;
    auto flush = [&](uint32_t g) {
        const ulonglong2 x0 = red_half[0], x1 = red_half[1], x2 = red_half[2], x3 = red_half[3];
        const float2 h = halves2(add2(add2(add2(x0.x, x0.y), add2(x1.x, x1.y)), add2(add2(x2.x, x2.y), add2(x3.x, x3.y))));
        float sum = h.x + h.y;
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (red_lane && g != kNone) atomicAdd(accum + (size_t)g * 16 + (lane >> 1), sum);
    };

    EntryFeed feed;
    feed.start(batch_ids(0), batch_ids(1), bounds);
    feed.stage(sm.stage[0], total, patch_x, patch_y, records, bounds, batch_ids(2), lane);
    for (int b = 0; b < n_batches; ++b) {
        const int32_t batch_end = top - 32 * b;
        const uint32_t staged = feed.mask;
        if (b + 1 < n_batches) {
            // (b + 1)'s buffer was last read before the walk of b - 1 ended
            __syncwarp();
            feed.stage(sm.stage[(b + 1) & 1], total - 32 * (b + 1), patch_x, patch_y, records, bounds, batch_ids(b + 3), lane);
            if (!staged) continue;
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        const WarpStage& st = sm.stage[b & 1];
        // entries whose forms miss this warp's patch are dropped up front
        bool reached = staged >> lane & 1u;
        if (reached) reached = patch_reached<MODEL>(st.rec[0][lane], st.rec[1][lane], st.rec[2][lane], st.zw[lane].x, rays);
        uint32_t bits = __ballot_sync(0xffffffffu, reached);
        while (bits) {
            const int t = __ffs(bits) - 1;
            bits &= bits - 1;
            // Every lane evaluates the pair (the record reads are warp-wide broadcasts); pixels that are outside
            // the image, beyond their last contributor or below the alpha threshold continue with alpha = vis = 0,
            // which makes every term they add exactly zero, so no per-lane branching is needed below.
            const float4 r0 = st.rec[0][t], r1 = st.rec[1][t], r2 = st.rec[2][t], r3 = st.rec[3][t];
            flush(pending);   // in the shadow of this entry's evaluation
            pending = kNone;
            const PixelForms<PX> f = pixel_forms<MODEL, PX>(r0, r1, r2, dx, dy, dz);
            float E[PX], limit[PX], den[PX], ex[PX], vis[PX], ov[PX], alpha[PX];
            P::get(f.E, E);
            P::get(mul2(P::all(r1.w), f.den), limit);
            P::get(f.den, den);
            bool valid[PX], any_valid = false, near_cut = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                valid[q] = batch_end - t <= bin_final[q] && E[q] <= limit[q];   // the forward's comparison: it decides for NaN too
                any_valid = any_valid || valid[q];
                den[q] = rcp_approx(den[q]);
            }
            const V rden = P::make(den), phi = mul2(f.E, rden);
            P::get(mul2(P::all(r0.w), phi), ex);
#pragma unroll
            for (int q = 0; q < PX; ++q) vis[q] = exp2_approx(ex[q]);
            P::get(mul2(P::all(r3.w), P::make(vis)), ov);
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                alpha[q] = fminf(0.999f, ov[q]);
                near_cut = near_cut || (valid[q] && alpha[q] < r2.w);
            }
            const uint32_t some = __ballot_sync(0xffffffffu, any_valid), ask = __ballot_sync(0xffffffffu, near_cut);
            if (!some) continue;
            if (ask) {
                const uint32_t kept = kept_at_cut<PX>(cuts + st.sid[t], n_cuts, &sm.ray[0][lane], 32, r3.w);
                any_valid = false;
#pragma unroll
                for (int q = 0; q < PX; ++q) {
                    valid[q] = valid[q] && ((kept >> q & 1u) || !(alpha[q] < r2.w));
                    any_valid = any_valid || valid[q];
                }
                if (!__any_sync(0xffffffffu, any_valid)) continue;
            }
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                if (!valid[q]) alpha[q] = 0.f;
                // geometry and opacity only while alpha is not clamped at 0.999
                if (!(valid[q] && ov[q] <= 0.999f)) vis[q] = 0.f;
            }
            const V al = P::make(alpha);
            // 1 / (1 - alpha), 1 - alpha in [0.001, 1]: the hardware estimate and one Newton step (relative error below 2^-23)
            const V na = add2(al, minus_one);
            float y0[PX];
            P::get(na, y0);
#pragma unroll
            for (int q = 0; q < PX; ++q) y0[q] = rcp_approx(-y0[q]);
            const V y = P::make(y0), ra = fma2(y, fma2(na, y, one), y);
            T = mul2(T, ra);
            const V fac = mul2(al, T), nfac = mul2(fac, minus_one);
            // minus colour . v_colour of this entry: the colours only ever meet the output gradient in this product
            V ncv = fma2(P::all(r3.x), vcr, fma2(P::all(r3.y), vcg, mul2(P::all(r3.z), vcb)));
            if (EXTRA) ncv = fma2(P::all(st.zw[t].y), vcx, ncv);
            const V v_alpha = fma2(ra, behind, mul2(mul2(ncv, minus_one), T));
            behind = fma2(ncv, fac, behind);
            const V q = mul2(P::make(vis), v_alpha);
            const V omega = mul2(f.w, rden), qo = mul2(q, omega);
            const V th1 = mul2(qo, f.e1), th2 = mul2(qo, f.e2), t1 = mul2(th1, omega), t2 = mul2(th2, omega);
            const uint32_t g = st.sid[t];
            auto put = [&](int k, V v) { sm.red[k * kRedStride + lane] = P::sum(v); };
            put(0, th1); put(1, th2); put(2, mul2(th1, phi)); put(3, mul2(th2, phi));
            put(4, mul2(t1, f.e1)); put(5, mul2(t1, f.e2)); put(6, mul2(t2, f.e2)); put(7, mul2(q, phi));
            put(8, mul2(nfac, vcr)); put(9, mul2(nfac, vcg)); put(10, mul2(nfac, vcb)); put(11, q);
            if (XGRAD) {
                const float s = __reduce_add_sync_f32(P::sum(mul2(nfac, vcx)));
                if (lane == 0) atomicAdd(accum_extra + g, s);
            }
            __syncwarp();
            pending = g;
        }
    }
    flush(pending);
}

// ---------------------------------------------------------------------------------------------
// Per-Gaussian gradient from the accumulated sums. Outputs gradients w.r.t. the ACTIVATED mean / quaternion / scale /
// opacity and the colour. `opacity` is the blended opacity of the record.
//
// One ray origin. With u' = O u (RayFrame) the loss reaches M and g through phi(u', g') and |g|^2 only, and
// v_M = sum v_u (x) d + v_g (x) (o - mu) collapses to O^T Y O S R^T with the symmetric Y below: the part of the two terms that
// grows with the distance cancels in the algebra instead of in float32. Then v_scale_j = -(O^T Y O)_jj / s_j and
// v_mean = -M^T v_g.
// ---------------------------------------------------------------------------------------------
struct GaussGrad {
    float v_mean[3], v_quat[4], v_scale[3], v_opac, v_rgb[3];
};

__device__ __forceinline__ void gaussian_vjp(const CamDev& cam, const float* acc /*16*/, f3 mean, float qw, float qx,
                                             float qy, float qz, f3 scale, float opacity, GaussGrad& o) {
    float R[9], inv_norm, qn[4];
    quat_to_rotmat_renorm(qw, qx, qy, qz, R, inv_norm, qn);
    const float is[3] = {1.0f / scale.x, 1.0f / scale.y, 1.0f / scale.z};
    const f3 om{cam.ro[0] - mean.x, cam.ro[1] - mean.y, cam.ro[2] - mean.z};
    float G[3], vMt[9];
    if (cam.rs_type == LFS_SHUTTER_GLOBAL && !cam.has_end) {
        RayFrame f;
        ray_frame(cam, R, om, scale, is, f);
        const float og = opacity * f.gamma, y = -og * f.gamma;
        const float Y00 = y * acc[4], Y01 = y * acc[5], Y11 = y * acc[6], Y02 = -y * acc[2], Y12 = -y * acc[3];
        const float Y22 = y * (acc[7] - acc[4] - acc[6]);
        const float g0 = -og * acc[0], g1 = -og * acc[1], g2 = og * acc[7];
        const float sc[3] = {scale.x, scale.y, scale.z};
        float YO[9], Z[9];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            YO[k] = Y00 * f.O[k] + Y01 * f.O[3 + k] + Y02 * f.O[6 + k];
            YO[3 + k] = Y01 * f.O[k] + Y11 * f.O[3 + k] + Y12 * f.O[6 + k];
            YO[6 + k] = Y02 * f.O[k] + Y12 * f.O[3 + k] + Y22 * f.O[6 + k];
            G[k] = f.O[k] * g0 + f.O[3 + k] * g1 + f.O[6 + k] * g2;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int k = 0; k < 3; ++k) Z[j * 3 + k] = (f.O[j] * YO[k] + f.O[3 + j] * YO[3 + k] + f.O[6 + j] * YO[6 + k]) * sc[k];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int a = 0; a < 3; ++a) vMt[j * 3 + a] = Z[j * 3] * R[a * 3] + Z[j * 3 + 1] * R[a * 3 + 1] + Z[j * 3 + 2] * R[a * 3 + 2];
            o.v_scale[j] = -is[j] * is[j] * Z[j * 3 + j];
        }
        o.v_rgb[0] = acc[8]; o.v_rgb[1] = acc[9]; o.v_rgb[2] = acc[10];
        o.v_opac = acc[11];
    } else {
        const float omu[3] = {om.x, om.y, om.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            G[a] = acc[9 + a];
#pragma unroll
            for (int b = 0; b < 3; ++b) vMt[a * 3 + b] = acc[a * 3 + b] + G[a] * omu[b];   // A + G (x) (o - mu)
        }
        // v_scale[j] = -is[j]^2 sum_a R[a][j] v_M[a][j] = -is[j]^2 sum_a R[a][j] vMt[j][a]
#pragma unroll
        for (int jx = 0; jx < 3; ++jx)
            o.v_scale[jx] = -is[jx] * is[jx] * (R[0 * 3 + jx] * vMt[jx * 3 + 0] + R[1 * 3 + jx] * vMt[jx * 3 + 1] + R[2 * 3 + jx] * vMt[jx * 3 + 2]);
        o.v_rgb[0] = acc[12]; o.v_rgb[1] = acc[13]; o.v_rgb[2] = acc[14];
        o.v_opac = acc[15];
    }
    // v_(o-mu) = Mt^T G with Mt[a][b] = is[a] R[b][a]  ->  sum_a is[a] R[b][a] G[a]
#pragma unroll
    for (int b = 0; b < 3; ++b)
        o.v_mean[b] = -(is[0] * R[b * 3 + 0] * G[0] + is[1] * R[b * 3 + 1] * G[1] + is[2] * R[b * 3 + 2] * G[2]);
    // v_R[a][b] = v_M[a][b] is[b] with v_M = v_Mt^T
    float vR[9];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) vR[a * 3 + b] = vMt[b * 3 + a] * is[b];
    const float w = qn[0], x = qn[1], y = qn[2], z = qn[3];
    const float vqn[4] = {
        2.f * (x * (vR[7] - vR[5]) + y * (vR[2] - vR[6]) + z * (vR[3] - vR[1])),
        2.f * (-2.f * x * (vR[4] + vR[8]) + y * (vR[3] + vR[1]) + z * (vR[6] + vR[2]) + w * (vR[7] - vR[5])),
        2.f * (x * (vR[3] + vR[1]) - 2.f * y * (vR[0] + vR[8]) + z * (vR[7] + vR[5]) + w * (vR[2] - vR[6])),
        2.f * (x * (vR[6] + vR[2]) + y * (vR[7] + vR[5]) - 2.f * z * (vR[0] + vR[4]) + w * (vR[3] - vR[1]))};
    const float dq = vqn[0] * qn[0] + vqn[1] * qn[1] + vqn[2] * qn[2] + vqn[3] * qn[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) o.v_quat[k] = (vqn[k] - dq * qn[k]) * inv_norm;
}

__global__ void __launch_bounds__(256) grad_epilogue_op_kernel(
    int N, const CamDev* __restrict__ cams, const float* __restrict__ accum, const float4* __restrict__ records,
    const float* __restrict__ means, const float* __restrict__ quats, const float* __restrict__ scales, int channels, const float* __restrict__ accum_extra,
    float* __restrict__ v_means, float* __restrict__ v_quats, float* __restrict__ v_scales, float* __restrict__ v_colors,
    float* __restrict__ v_opacities) {
    const CamDev& cam = cams[0];
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < N; g += gridDim.x * blockDim.x) {
        float acc[16];
        const float4* a4 = reinterpret_cast<const float4*>(accum) + (size_t)g * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float4 t = a4[k]; acc[k * 4] = t.x; acc[k * 4 + 1] = t.y; acc[k * 4 + 2] = t.z; acc[k * 4 + 3] = t.w; }
        const float4 q = reinterpret_cast<const float4*>(quats)[g];
        GaussGrad o;
        gaussian_vjp(cam, acc, f3{means[g * 3], means[g * 3 + 1], means[g * 3 + 2]}, q.x, q.y, q.z, q.w,
                     f3{scales[g * 3], scales[g * 3 + 1], scales[g * 3 + 2]}, records[(size_t)g * 4 + 3].w, o);
#pragma unroll
        for (int k = 0; k < 3; ++k) { v_means[g * 3 + k] = o.v_mean[k]; v_scales[g * 3 + k] = o.v_scale[k]; }
        if (channels >= 3) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v_colors[(size_t)g * channels + k] = o.v_rgb[k];
        }
        if (channels != 3) v_colors[(size_t)g * channels + channels - 1] = accum_extra[g];
#pragma unroll
        for (int k = 0; k < 4; ++k) v_quats[g * 4 + k] = o.v_quat[k];
        v_opacities[g] = o.v_opac;
    }
}

__device__ __forceinline__ void adam_small_update(float& p, float& m, float& v, float g, float step_size, const AdamSmall& A) {
    const float m1 = A.beta1 * m + (1.0f - A.beta1) * g;
    const float m2 = A.beta2 * v + (1.0f - A.beta2) * g * g;
    const float denom = sqrtf(m2) * A.bc2_sqrt_rcp + A.eps;
    p -= step_size * m1 / denom;
    m = m1;
    v = m2;
}
// One row of W floats of small group `gi` (index into AdamSmall): p_in are the parameter values already in registers.
template <int W>
__device__ __forceinline__ void adam_small_row(const AdamSmall& A, int gi, size_t row, const float* p_in, const float* grad) {
    float* mm = A.m[gi] + row * W;
    float* vv = A.v[gi] + row * W;
    float* pp = A.p[gi] + row * W;
    float p[W], m[W], v[W];
#pragma unroll
    for (int k = 0; k < W; ++k) { p[k] = p_in[k]; m[k] = mm[k]; v[k] = vv[k]; }
#pragma unroll
    for (int k = 0; k < W; ++k) adam_small_update(p[k], m[k], v[k], grad[k] * A.grad_scale, A.step_size[gi], A);
#pragma unroll
    for (int k = 0; k < W; ++k) { pp[k] = p[k]; mm[k] = m[k]; vv[k] = v[k]; }
}

// Fused-path epilogue: raw-parameter gradients (activation backward folded in) and the SH backward.
// Each warp handles 32 consecutive Gaussians per iteration; their shN gradient rows (the bulk of the
// output, (K-1)*3 floats each) are staged in shared memory and written as one contiguous run.
// ADAM: the five small groups (means, sh0, scales, rotations, opacities) are not written as gradients but applied at
// once, in place, with the moments in A (the parameter pointers below alias A.p, hence no __restrict__ on them); the
// shN gradient leaves as its two rank-1 factors (sh_factors) for adam_sh_rank1_kernel.
// ROWS: the shN gradient leaves as rows; without them the kernel neither holds their staging nor the registers of its stores.
template <bool ADAM, bool ROWS>
__global__ void __launch_bounds__(256, ROWS ? 3 : 4) grad_epilogue_fused_kernel(
    int N, int K, int sh_degree, const CamDev* __restrict__ cams, const float* accum /* ADAM: aliased by g_shN */,
    const float4* __restrict__ records, const int32_t* __restrict__ radii,
    const float* means, const float* sh0, const float* scaling_raw, const float* rotation_raw, const float* opacity_raw,
    float* __restrict__ g_means, float* __restrict__ g_sh0, float* g_shN, float* __restrict__ g_scaling,
    float* __restrict__ g_rotation, float* __restrict__ g_opacity, int accumulate, float scaling_modifier, int sh_factors,
    AdamSmall A) {
    extern __shared__ __align__(16) float s_rows[];
    const bool rows_aligned = (reinterpret_cast<uintptr_t>(g_shN) & 15) == 0;
    const CamDev& cam = cams[0];
    const int rest = (K - 1) * 3;
    const int nb = (sh_degree + 1) * (sh_degree + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my = s_rows + (size_t)warp * 32 * rest;
    const int n_chunks = (N + 31) / 32;
    const int warps_total = gridDim.x * (blockDim.x >> 5);
    for (int chunk = blockIdx.x * (blockDim.x >> 5) + warp; chunk < n_chunks; chunk += warps_total) {
        const int g = chunk * 32 + lane;
        const bool in_range = g < N;
        // Everything a visible Gaussian needs is requested together with its radii (one round trip to memory instead of
        // two); for the others the values are dropped.
        int2 rad = make_int2(0, 0);
        float4 a_in[4], qr = make_float4(1.f, 0.f, 0.f, 0.f), r3 = make_float4(0.f, 0.f, 0.f, 0.f);
        float m_in[3] = {0.f, 0.f, 0.f}, s_in[3] = {0.f, 0.f, 0.f}, o_in = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) a_in[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in_range) {
            rad = reinterpret_cast<const int2*>(radii)[g];
            if (rad.x > 0 && rad.y > 0) {   // culled Gaussians have no accumulator row: the projection zeroes visible rows only
                const float4* a4 = reinterpret_cast<const float4*>(accum) + (size_t)g * 4;
#pragma unroll
                for (int k = 0; k < 4; ++k) a_in[k] = a4[k];
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) { m_in[k] = means[g * 3 + k]; s_in[k] = scaling_raw[g * 3 + k]; }
            o_in = opacity_raw[g];
            qr = reinterpret_cast<const float4*>(rotation_raw)[g];
            r3 = records[(size_t)g * 4 + 3];
        }
        const bool visible = in_range && rad.x > 0 && rad.y > 0;
        float gm[3] = {0.f, 0.f, 0.f}, g0[3] = {0.f, 0.f, 0.f}, gs[3] = {0.f, 0.f, 0.f}, gq[4] = {0.f, 0.f, 0.f, 0.f}, go = 0.f;
        float vc[3] = {0.f, 0.f, 0.f};
        float B[25];
#pragma unroll
        for (int k = 0; k < 25; ++k) B[k] = 0.f;
        if (visible) {
            float acc[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) { const float4 t = a_in[k]; acc[k * 4] = t.x; acc[k * 4 + 1] = t.y; acc[k * 4 + 2] = t.z; acc[k * 4 + 3] = t.w; }
            const f3 mean{m_in[0], m_in[1], m_in[2]};
            const float opacity = (float)(1.0 / (1.0 + exp(-(double)o_in)));
            // scale as blended: exp(raw) * modifier; d(scale)/d(raw) is the same product
            f3 scale{(float)exp((double)s_in[0]), (float)exp((double)s_in[1]), (float)exp((double)s_in[2])};
            if (scaling_modifier != 1.0f) { scale.x *= scaling_modifier; scale.y *= scaling_modifier; scale.z *= scaling_modifier; }
            const float n2 = ((qr.x * qr.x + qr.y * qr.y) + qr.z * qr.z) + qr.w * qr.w;
            const float nrm = fmaxf(sqrtf(n2), 1e-12f);
            const float q[4] = {qr.x / nrm, qr.y / nrm, qr.z / nrm, qr.w / nrm};
            GaussGrad o;
            gaussian_vjp(cam, acc, mean, q[0], q[1], q[2], q[3], scale, r3.w, o);
            // activation backward: sigmoid, exp, x / max(|x|, eps)
            go = o.v_opac * (opacity * (1.0f - opacity));
            gs[0] = o.v_scale[0] * scale.x; gs[1] = o.v_scale[1] * scale.y; gs[2] = o.v_scale[2] * scale.z;
            const float dq = o.v_quat[0] * q[0] + o.v_quat[1] * q[1] + o.v_quat[2] * q[2] + o.v_quat[3] * q[3];
#pragma unroll
            for (int k = 0; k < 4; ++k) gq[k] = (o.v_quat[k] - q[k] * dq) / nrm;
#pragma unroll
            for (int k = 0; k < 3; ++k) gm[k] = o.v_mean[k];
            // colour clamp mask, then SH backward
            vc[0] = r3.x <= 0.f ? 0.f : o.v_rgb[0];
            vc[1] = r3.y <= 0.f ? 0.f : o.v_rgb[1];
            vc[2] = r3.z <= 0.f ? 0.f : o.v_rgb[2];
            sh_basis(sh_degree, mean.x - cam.campos[0], mean.y - cam.campos[1], mean.z - cam.campos[2], B);
#pragma unroll
            for (int k = 0; k < 3; ++k) g0[k] = B[0] * vc[k];
        }
        if (!ROWS && g_shN && sh_factors) {
            // the two factors of the rank-1 rows instead of the rows: [N,6] = (clamped colour gradient, unit view direction)
            // at the start of the shN gradient tensor, for the data-parallel exchange that sums the outer products
            if (in_range) {
                float dx = 0.f, dy = 0.f, dz = 0.f;
                if (visible) {
                    dx = m_in[0] - cam.campos[0]; dy = m_in[1] - cam.campos[1]; dz = m_in[2] - cam.campos[2];
                    const float inorm = rsqrtf(dx * dx + dy * dy + dz * dz);
                    dx *= inorm; dy *= inorm; dz *= inorm;
                }
                // ADAM: the factors go into the Gaussian's own (now consumed) row of 16 sums
                float2* f = ADAM ? reinterpret_cast<float2*>(g_shN) + (size_t)g * 8 : reinterpret_cast<float2*>(g_shN) + (size_t)g * 3;
                f[0] = make_float2(vc[0], vc[1]); f[1] = make_float2(vc[2], dx); f[2] = make_float2(dy, dz);
            }
        } else if (ROWS) {  // otherwise the caller forms these rows itself from the sh0 gradient (adam_sh_rank1_kernel)
            for (int k = 1; k < K; ++k) {
                const float w = k < nb ? B[k] : 0.f;
#pragma unroll
                for (int c = 0; c < 3; ++c) my[lane * rest + (k - 1) * 3 + c] = w * vc[c];
            }
            __syncwarp();
            const int n_rows = min(32, N - chunk * 32);
            const int total = n_rows * rest;
            float* dst = g_shN + (size_t)chunk * 32 * rest;
            if (!accumulate || __any_sync(0xffffffffu, visible)) store_rows(dst, my, total, lane, rows_aligned, accumulate != 0);
            __syncwarp();
        }
        if (ADAM) {
            if (in_range) {
                const float c_in[3] = {sh0[g * 3], sh0[g * 3 + 1], sh0[g * 3 + 2]};
                const float q_in[4] = {qr.x, qr.y, qr.z, qr.w};
                adam_small_row<3>(A, 0, (size_t)g, m_in, gm);
                adam_small_row<3>(A, 1, (size_t)g, c_in, g0);
                adam_small_row<3>(A, 2, (size_t)g, s_in, gs);
                adam_small_row<4>(A, 3, (size_t)g, q_in, gq);
                adam_small_row<1>(A, 4, (size_t)g, &o_in, &go);
            }
        } else if (in_range && (visible || !accumulate)) {
            if (accumulate) {
#pragma unroll
                for (int k = 0; k < 3; ++k) { g_means[g * 3 + k] += gm[k]; g_sh0[g * 3 + k] += g0[k]; g_scaling[g * 3 + k] += gs[k]; }
#pragma unroll
                for (int k = 0; k < 4; ++k) g_rotation[g * 4 + k] += gq[k];
                g_opacity[g] += go;
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) { g_means[g * 3 + k] = gm[k]; g_sh0[g * 3 + k] = g0[k]; g_scaling[g * 3 + k] = gs[k]; }
                reinterpret_cast<float4*>(g_rotation)[g] = make_float4(gq[0], gq[1], gq[2], gq[3]);
                g_opacity[g] = go;
            }
        }
    }
}

// Adam on the higher-order SH coefficients without a gradient tensor. For one camera the gradient row of a Gaussian
// is the outer product of the SH basis of its view direction with the clamped colour gradient vc, and the sh0
// gradient already holds Y00 * vc; so the rows are rebuilt here, 32 Gaussians per warp in shared memory, and the
// parameter / moment rows (one contiguous run per warp) are streamed through once, 16 bytes per lane and U vectors of
// each tensor in flight. Same update arithmetic as the optimizer kernels.
__device__ __forceinline__ void adam_rank1_update(float& p, float& m, float& v, float g, const AdamRank1& A) {
    const float m1 = A.beta1 * m + (1.0f - A.beta1) * g;
    const float m2 = A.beta2 * v + (1.0f - A.beta2) * g * g;
    const float denom = sqrtf(m2) * A.bc2_sqrt_rcp + A.eps;
    p -= A.step_size * m1 / denom;
    m = m1;
    v = m2;
}
// KT: the number of SH coefficients when known at compile time (16 = degree 3, the training default; the row loop
// then unrolls and the basis stays in registers), 0 = generic.
template <int KT>
__global__ void __launch_bounds__(256, 4) adam_sh_rank1_kernel(int N, int K_rt, int sh_degree, const float* __restrict__ campos,
                                                               const float* __restrict__ means, const float* __restrict__ g_sh0,
                                                               const float* __restrict__ factors, int factor_stride, AdamRank1 A) {
    extern __shared__ __align__(16) float s_rows[];
    constexpr int U = 3;
    const int K = KT ? KT : K_rt;
    float cx = 0.f, cy = 0.f, cz = 0.f;
    if (!factors) { cx = campos[0]; cy = campos[1]; cz = campos[2]; }
    const int rest = (K - 1) * 3;
    const int nb = (sh_degree + 1) * (sh_degree + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my = s_rows + (size_t)warp * 32 * rest;
    const int n_chunks = (N + 31) / 32;
    const int warps_total = gridDim.x * (blockDim.x >> 5);
    for (int chunk = blockIdx.x * (blockDim.x >> 5) + warp; chunk < n_chunks; chunk += warps_total) {
        const int g = chunk * 32 + lane;
        float vc[3] = {0.f, 0.f, 0.f}, dir[3] = {0.f, 0.f, 0.f};
        if (g < N) {
            if (factors) {
                // written by the gradient stage: (clamped colour gradient, unit view direction)
                const float2* f = reinterpret_cast<const float2*>(factors + (size_t)g * factor_stride);
                const float2 f0 = f[0], f1 = f[1], f2 = f[2];
                vc[0] = f0.x; vc[1] = f0.y; vc[2] = f1.x; dir[0] = f1.y; dir[1] = f2.x; dir[2] = f2.y;
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) vc[c] = g_sh0[g * 3 + c] / 0.2820947917738781f;
            }
        }
        float B[25];
#pragma unroll
        for (int k = 0; k < 25; ++k) B[k] = 0.f;
        if (vc[0] != 0.f || vc[1] != 0.f || vc[2] != 0.f) {
            if (!factors) { dir[0] = means[g * 3] - cx; dir[1] = means[g * 3 + 1] - cy; dir[2] = means[g * 3 + 2] - cz; }
            sh_basis(sh_degree, dir[0], dir[1], dir[2], B);
        }
        if (KT) {
#pragma unroll
            for (int k = 1; k < (KT ? KT : 1); ++k) {
                const float w = k < nb ? B[k] : 0.f;
#pragma unroll
                for (int c = 0; c < 3; ++c) my[lane * rest + (k - 1) * 3 + c] = w * vc[c];
            }
        } else {
            for (int k = 1; k < K; ++k) {
                const float w = k < nb ? B[k] : 0.f;
#pragma unroll
                for (int c = 0; c < 3; ++c) my[lane * rest + (k - 1) * 3 + c] = w * vc[c];
            }
        }
        __syncwarp();
        const int total = min(32, N - chunk * 32) * rest;
        const size_t base = (size_t)chunk * 32 * rest;
        float* __restrict__ pp = A.p + base;
        float* __restrict__ mm = A.m + base;
        float* __restrict__ vv = A.v + base;
        int done = 0;
        if (A.vec) {
            const int total4 = total >> 2;
            float4* __restrict__ p4 = reinterpret_cast<float4*>(pp);
            float4* __restrict__ m4 = reinterpret_cast<float4*>(mm);
            float4* __restrict__ v4 = reinterpret_cast<float4*>(vv);
            const float4* __restrict__ g4 = reinterpret_cast<const float4*>(my);
            for (int i0 = lane; i0 < total4; i0 += 32 * U) {
                float4 p[U], m[U], v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + 32 * u;
                    if (i < total4) { p[u] = p4[i]; m[u] = m4[i]; v[u] = v4[i]; }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + 32 * u;
                    if (i < total4) {
                        const float4 gr = g4[i];
                        adam_rank1_update(p[u].x, m[u].x, v[u].x, gr.x * A.grad_scale, A);
                        adam_rank1_update(p[u].y, m[u].y, v[u].y, gr.y * A.grad_scale, A);
                        adam_rank1_update(p[u].z, m[u].z, v[u].z, gr.z * A.grad_scale, A);
                        adam_rank1_update(p[u].w, m[u].w, v[u].w, gr.w * A.grad_scale, A);
                        p4[i] = p[u]; m4[i] = m[u]; v4[i] = v[u];
                    }
                }
            }
            done = total4 << 2;
        }
        for (int i = done + lane; i < total; i += 32) {
            float p = pp[i], m = mm[i], v = vv[i];
            adam_rank1_update(p, m, v, my[i] * A.grad_scale, A);
            pp[i] = p; mm[i] = m; vv[i] = v;
        }
        __syncwarp();
    }
}

// Data-parallel form of adam_sh_rank1_kernel: this rank owns the elements [lo, lo + n) of the shN tensor. For the rows
// that intersect them, the gradient row is the sum over ranks of (SH basis of that rank's view direction) x (that
// rank's clamped colour gradient), both read from the rank's factor buffer [N,6] through its peer pointer (24 bytes per
// row and rank instead of the 12 (K-1) bytes of a materialised row); then Adam with the shard-local moments and 16-byte
// stores of the new coefficients into every rank's parameter buffer (plain peer stores, or one multimem.st through the
// NVSwitch multicast address of the tensor). Plain peer loads; the caller orders the launch against the other ranks.
template <int KT>
__global__ void __launch_bounds__(256) dp_sh_rank1_kernel(int K_rt, int sh_degree, DpRank1 A) {
    extern __shared__ __align__(16) float s_rows[];
    constexpr int U = 2;
    constexpr int kPre = 4;
    const int K = KT ? KT : K_rt;
    const int rest = (K - 1) * 3;
    const int nb = (sh_degree + 1) * (sh_degree + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my = s_rows + (size_t)warp * 32 * rest;
    const int64_t hi = A.lo + A.n;
    const int64_t chunk_elems = (int64_t)32 * rest;
    const int64_t first_chunk = A.lo / chunk_elems, last_chunk = (hi - 1) / chunk_elems;
    const int warps_total = gridDim.x * (blockDim.x >> 5);
    for (int64_t chunk = first_chunk + blockIdx.x * (blockDim.x >> 5) + warp; chunk <= last_chunk; chunk += warps_total) {
        const int64_t g = chunk * 32 + lane;
        for (int j = 0; j < rest; ++j) my[lane * rest + j] = 0.f;
        if (g < A.N) {
            // kPre ranks' factors are in flight at a time (a peer load takes microseconds)
            for (int r0 = 0; r0 < A.world; r0 += kPre) {
                float2 F[kPre][3];
#pragma unroll
                for (int q = 0; q < kPre; ++q) {
                    if (r0 + q < A.world) {
                        const float2* f = reinterpret_cast<const float2*>(A.factors[r0 + q]) + g * 3;
                        F[q][0] = f[0]; F[q][1] = f[1]; F[q][2] = f[2];
                    } else {
                        F[q][0] = F[q][1] = F[q][2] = make_float2(0.f, 0.f);
                    }
                }
#pragma unroll
                for (int q = 0; q < kPre; ++q) {
                    const float vc[3] = {F[q][0].x, F[q][0].y, F[q][1].x};
                    if (vc[0] == 0.f && vc[1] == 0.f && vc[2] == 0.f) continue;
                    float B[25];
#pragma unroll
                    for (int k = 0; k < 25; ++k) B[k] = 0.f;
                    sh_basis(sh_degree, F[q][1].y, F[q][2].x, F[q][2].y, B);
                    if (KT) {
#pragma unroll
                        for (int k = 1; k < (KT ? KT : 1); ++k) {
                            const float w = k < nb ? B[k] : 0.f;
#pragma unroll
                            for (int c = 0; c < 3; ++c) my[lane * rest + (k - 1) * 3 + c] += w * vc[c];
                        }
                    } else {
                        for (int k = 1; k < K; ++k) {
                            const float w = k < nb ? B[k] : 0.f;
#pragma unroll
                            for (int c = 0; c < 3; ++c) my[lane * rest + (k - 1) * 3 + c] += w * vc[c];
                        }
                    }
                }
            }
        }
        __syncwarp();
        const int64_t c0 = chunk * chunk_elems;
        const int64_t e0 = max(A.lo, c0), e1 = min(hi, c0 + chunk_elems);
        const int total = (int)(e1 - e0);
        const float* __restrict__ grad = my + (e0 - c0);
        const float* __restrict__ pp = A.shN[0] + e0;   // every rank holds the same coefficients; read the local copy
        float* __restrict__ mm = A.m + (e0 - A.lo);
        float* __restrict__ vv = A.v + (e0 - A.lo);
        int done = 0;
        if (A.vec) {
            const int total4 = total >> 2;
            const float4* __restrict__ p4 = reinterpret_cast<const float4*>(pp);
            float4* __restrict__ m4 = reinterpret_cast<float4*>(mm);
            float4* __restrict__ v4 = reinterpret_cast<float4*>(vv);
            const float4* __restrict__ g4 = reinterpret_cast<const float4*>(grad);
            for (int i0 = lane; i0 < total4; i0 += 32 * U) {
                float4 p[U], m[U], v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + 32 * u;
                    if (i < total4) { p[u] = p4[i]; m[u] = m4[i]; v[u] = v4[i]; }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + 32 * u;
                    if (i < total4) {
                        const float4 gr = g4[i];
                        adam_rank1_update(p[u].x, m[u].x, v[u].x, gr.x * A.adam.grad_scale, A.adam);
                        adam_rank1_update(p[u].y, m[u].y, v[u].y, gr.y * A.adam.grad_scale, A.adam);
                        adam_rank1_update(p[u].z, m[u].z, v[u].z, gr.z * A.adam.grad_scale, A.adam);
                        adam_rank1_update(p[u].w, m[u].w, v[u].w, gr.w * A.adam.grad_scale, A.adam);
                        m4[i] = m[u]; v4[i] = v[u];
                        if (A.mc_shN) {
                            multimem_st4(A.mc_shN + e0 + 4 * (int64_t)i, p[u]);
                        } else {
                            for (int r = 0; r < A.world; ++r) reinterpret_cast<float4*>(A.shN[r] + e0)[i] = p[u];
                        }
                    }
                }
            }
            done = total4 << 2;
        }
        for (int i = done + lane; i < total; i += 32) {
            float p = pp[i], m = mm[i], v = vv[i];
            adam_rank1_update(p, m, v, grad[i] * A.adam.grad_scale, A.adam);
            mm[i] = m; vv[i] = v;
            if (A.mc_shN) {
                multimem_st1(A.mc_shN + e0 + i, p);
            } else {
                for (int r = 0; r < A.world; ++r) A.shN[r][e0 + i] = p;
            }
        }
        __syncwarp();
    }
}

}  // namespace

int launch_raster_fwd(const RasterArgs& a, float* render, float* alphas, int32_t* last_ids, float* extra_sum, cudaStream_t st) {
    const int n_tiles = a.tw * a.th;
    if (n_tiles == 0) return LFS_OK;
    if (a.channels != 1 && a.channels != 3 && a.channels != 4) { set_error("raster_fwd: channels must be 1, 3 or 4"); return LFS_EINVAL; }
    LFS_TIMED("raster_fwd", st);
    // Two pixels per thread where the patches of twice the size still fill the GPU. fwd us with one and two, 1296x840-like scenes of 100 k Gaussians: 510
    // tiles 91 and 117, 920 tiles 98 and 104, 1,400 tiles 122 and 107, 2,170 tiles 158 and 129. A fisheye shows the scene on a tenth of its tiles or
    // so: 600 k, 4,096 tiles 239 and 344, 8,100 tiles 216 and 278, 14,400 tiles 309 and 271. An equirectangular camera sees all around: 100 k and 600 k, 512
    // tiles 68 and 81, 91 and 100, 2,048 tiles 131 and 110, 125 and 106, 8,192 tiles 416 and 303, 381 and 276.
    const bool two = n_tiles >= (a.model == LFS_FISHEYE ? 80 : 8) * num_sms();
    const Outsized out = outsized_lists(a.tile_order, n_tiles);
#define LFS_FWD_RS(MODEL, EXTRA)                                                                                                    \
    raster_fwd_rs_kernel<MODEL, EXTRA><<<n_tiles, kBlock, 0, st>>>(a.cam, a.records, a.bounds, a.flatten_ids, a.tile_offsets, a.n_isects_dev,       \
                                                                   a.n_isects_host, a.overflow, a.background, a.masks, a.tile_order, a.channels,   \
                                                                   a.normalize, a.W, a.H, a.tw, n_tiles, render, alphas, last_ids, extra_sum)
#define LFS_FWD_PATCH(LAUNCH, MODEL, EXTRA, PX, VOTE, TILES, OUT)                                                                   \
    LAUNCH(raster_fwd_patch_kernel<MODEL, EXTRA, PX, VOTE>, (TILES) * (2 / PX), 128, 4 * sizeof(FwdPatchWarp<PX>), st,              \
        a.cam, a.records, a.cuts, a.n_cuts, a.bounds, a.flatten_ids, a.tile_offsets, a.n_isects_dev, a.n_isects_host, a.overflow, a.background,  \
        a.masks, a.tile_order, a.channels, a.normalize, a.W, a.H, a.tw, n_tiles, OUT, render, alphas, last_ids, extra_sum)
#define LFS_FWD2(MODEL, EXTRA)                                                                                                      \
    do {                                                                                                                            \
        constexpr bool kWide = MODEL != LFS_PINHOLE && MODEL != LFS_PINHOLE_OPENCV;                                                 \
        if (!two) { LFS_FWD_PATCH(launch, MODEL, EXTRA, 1, kWide, n_tiles, Outsized{}); break; }                                    \
        if (!out.share) { LFS_FWD_PATCH(launch, MODEL, EXTRA, 2, kWide, n_tiles, out); break; }                                     \
        LFS_FWD_PATCH(launch, MODEL, EXTRA, 1, true, out.slots, out);                                                               \
        LFS_FWD_PATCH(launch_beside, MODEL, EXTRA, 2, kWide, n_tiles, out);                                                         \
    } while (0)
#define LFS_FWD(MODEL) do { if (a.rolling) { if (extra) LFS_FWD_RS(MODEL, true); else LFS_FWD_RS(MODEL, false); }                   \
                            else if (extra) LFS_FWD2(MODEL, true); else LFS_FWD2(MODEL, false); } while (0)
    const bool extra = a.channels != 3;
    if (a.model == LFS_PINHOLE) LFS_FWD(LFS_PINHOLE);
    else if (a.model == LFS_PINHOLE_OPENCV) LFS_FWD(LFS_PINHOLE_OPENCV);
    else if (a.model == LFS_EQUIRECTANGULAR) { if (extra) LFS_FWD2(LFS_EQUIRECTANGULAR, true); else LFS_FWD2(LFS_EQUIRECTANGULAR, false); }
    else LFS_FWD(LFS_FISHEYE);
#undef LFS_FWD
#undef LFS_FWD2
#undef LFS_FWD_PATCH
#undef LFS_FWD_RS
    return check_launch("raster_fwd");
}

int launch_raster_bwd(const RasterArgs& a, const float* render_alphas, const int32_t* last_ids, const float* extra_sum,
                      const float* v_render, const float* v_alphas, float* accum, float* accum_extra, cudaStream_t st) {
    const int n_tiles = a.tw * a.th;
    if (n_tiles == 0) return LFS_OK;
    if (a.channels != 1 && a.channels != 3 && a.channels != 4) { set_error("raster_bwd: channels must be 1, 3 or 4"); return LFS_EINVAL; }
    if (a.normalize && !extra_sum) { set_error("raster_bwd: expected-depth modes need the forward's blended sum"); return LFS_EINVAL; }
    LFS_TIMED("raster_bwd", st);
    // Two pixels per thread where the patches of twice the size still fill the GPU (launch_raster_fwd). bwd us with one and two, planar, 100 k Gaussians: 256
    // tiles 190 and 266, 510 tiles 176 and 174 (20 k: 100 and 111, 400 k: 234 and 246), 920 tiles 211 and 165, 2,170 tiles 361 and 255; fisheye, 600 k: 4,096 tiles
    // 395 and 453, 8,100 tiles 418 and 379; equirectangular, 100 k and 600 k: 512 tiles 103 and 108, 102 and 116, 2,048 tiles 239 and 179, 204 and 155, 8,192 tiles
    // 756 and 519, 649 and 447.
    const bool extra = a.channels != 3, xgrad = extra && accum_extra != nullptr;
    const bool two = n_tiles >= (a.model == LFS_FISHEYE ? 40 : 4) * num_sms();
    const Outsized out = outsized_lists(a.tile_order, n_tiles);
#define LFS_BWD_RS(MODEL, EXTRA, XGRAD)                                                                                        \
    do {                                                                                                                       \
        constexpr int smem = (int)sizeof(BwdShared<64>);                                                                       \
        raster_bwd_rs_kernel<MODEL, 64, EXTRA, XGRAD><<<n_tiles, kBlock, smem, st>>>(                                          \
            a.cam, a.records, a.bounds, a.flatten_ids, a.tile_offsets, a.n_isects_dev, a.n_isects_host, a.overflow, a.background, \
            a.masks, a.tile_order, a.channels, a.normalize, a.W, a.H, a.tw, n_tiles, render_alphas, last_ids, extra_sum, v_render, \
            v_alphas, accum, accum_extra);                                                                                     \
    } while (0)
#define LFS_BWD_PATCH(LAUNCH, MODEL, EXTRA, XGRAD, PX, TILES, OUT)                                                             \
    do {                                                                                                                       \
        LAUNCH(raster_bwd_patch_kernel<MODEL, EXTRA, XGRAD, PX>, (TILES) * (2 / PX), 128, 4 * sizeof(BwdPatchWarp<PX>), st,    \
            a.cam, a.records, a.cuts, a.n_cuts, a.bounds, a.flatten_ids, a.tile_offsets, a.n_isects_dev, a.n_isects_host, a.overflow,    \
            a.background,                                                                                                      \
            a.masks, a.tile_order, a.channels, a.normalize, a.W, a.H, a.tw, n_tiles, OUT, render_alphas, last_ids, extra_sum, v_render, \
            v_alphas, accum, accum_extra);                                                                                     \
    } while (0)
#define LFS_BWD_ORIGIN(MODEL, EXTRA, XGRAD)                                                                                    \
    do {                                                                                                                       \
        if (!two) { LFS_BWD_PATCH(launch, MODEL, EXTRA, XGRAD, 1, n_tiles, Outsized{}); break; }                               \
        if (!out.share) { LFS_BWD_PATCH(launch, MODEL, EXTRA, XGRAD, 2, n_tiles, out); break; }                                \
        LFS_BWD_PATCH(launch, MODEL, EXTRA, XGRAD, 1, out.slots, out);                                                         \
        LFS_BWD_PATCH(launch_beside, MODEL, EXTRA, XGRAD, 2, n_tiles, out);                                                    \
    } while (0)
#define LFS_BWD_ANY(MODEL, EXTRA, XGRAD) do { if (a.rolling) LFS_BWD_RS(MODEL, EXTRA, XGRAD); else LFS_BWD_ORIGIN(MODEL, EXTRA, XGRAD); } while (0)
#define LFS_BWD(KIND, MODEL)                                                                                                   \
    do { if (!extra) KIND(MODEL, false, false); else if (!xgrad) KIND(MODEL, true, false); else KIND(MODEL, true, true); } while (0)
    if (a.model == LFS_PINHOLE) LFS_BWD(LFS_BWD_ANY, LFS_PINHOLE);
    else if (a.model == LFS_PINHOLE_OPENCV) LFS_BWD(LFS_BWD_ANY, LFS_PINHOLE_OPENCV);
    else if (a.model == LFS_EQUIRECTANGULAR) LFS_BWD(LFS_BWD_ORIGIN, LFS_EQUIRECTANGULAR);
    else LFS_BWD(LFS_BWD_ANY, LFS_FISHEYE);
#undef LFS_BWD
#undef LFS_BWD_ANY
#undef LFS_BWD_ORIGIN
#undef LFS_BWD_PATCH
#undef LFS_BWD_RS
    return check_launch("raster_bwd");
}

int launch_grad_epilogue_op(int N, const CamDev* cam, const float* accum, const float4* records, const float* means,
                            const float* quats, const float* scales, int channels, const float* accum_extra, float* v_means, float* v_quats,
                            float* v_scales, float* v_colors, float* v_opacities, cudaStream_t st) {
    if (N == 0) return LFS_OK;
    LFS_TIMED("grad_epilogue", st);
    grad_epilogue_op_kernel<<<grid_for(N, 256), 256, 0, st>>>(N, cam, accum, records, means, quats, scales, channels, accum_extra,
                                                              v_means, v_quats, v_scales, v_colors, v_opacities);
    return check_launch("grad_epilogue_op");
}

int launch_grad_epilogue_fused(int N, int K, int sh_degree, const CamDev* cam, const float* accum,
                               const float4* records, const int32_t* radii, const lfs_splats& p, const lfs_splats& g,
                               int accumulate, float scaling_modifier, int sh_factors, cudaStream_t st, const AdamSmall* adam) {
    if (N == 0) return LFS_OK;
    LFS_TIMED(adam ? "grad_epilogue_adam" : "grad_epilogue", st);
    const bool rows = !adam && g.shN && !sh_factors;
    const size_t row_bytes = (size_t)8 * 32 * (K - 1) * 3 * sizeof(float), smem = rows ? row_bytes : 0;
    if (row_bytes > 200 * 1024) { set_error("grad_epilogue_fused: too many SH coefficients"); return LFS_EINVAL; }
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(grad_epilogue_fused_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (adam) {
        grad_epilogue_fused_kernel<true, false><<<grid_for(N, 256), 256, 0, st>>>(
            N, K, sh_degree, cam, accum, records, radii, p.means, p.sh0, p.scaling_raw, p.rotation_raw, p.opacity_raw, nullptr,
            nullptr, const_cast<float*>(accum), nullptr, nullptr, nullptr, 0, scaling_modifier, 1, *adam);
    } else {
#define LFS_EPILOGUE(ROWS)                                                                                                          \
    grad_epilogue_fused_kernel<false, ROWS><<<grid_for(N, 256), 256, smem, st>>>(                                                   \
        N, K, sh_degree, cam, accum, records, radii, p.means, p.sh0, p.scaling_raw, p.rotation_raw, p.opacity_raw, g.means, g.sh0,  \
        g.shN, g.scaling_raw, g.rotation_raw, g.opacity_raw, accumulate, scaling_modifier, sh_factors, AdamSmall{})
        if (rows) LFS_EPILOGUE(true); else LFS_EPILOGUE(false);
#undef LFS_EPILOGUE
    }
    return check_launch("grad_epilogue_fused");
}

int launch_adam_sh_rank1(int N, int K, int sh_degree, const float* campos, const float* means, const float* g_sh0, float* p,
                         float* m, float* v, float step_size, float beta1, float beta2, float eps, float bc2_sqrt_rcp,
                         float grad_scale, cudaStream_t st, const float* factors, int factor_stride) {
    if (N == 0 || K <= 1) return LFS_OK;
    LFS_TIMED("adam_sh_rank1", st);
    const size_t smem = (size_t)8 * 32 * (K - 1) * 3 * sizeof(float);
    if (smem > 200 * 1024) { set_error("adam_sh_rank1: too many SH coefficients"); return LFS_EINVAL; }
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(adam_sh_rank1_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    AdamRank1 A{p, m, v, step_size, beta1, beta2, eps, bc2_sqrt_rcp, grad_scale,
                (int)(((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15) == 0)};
    if (K == 16) adam_sh_rank1_kernel<16><<<grid_for(N, 256), 256, smem, st>>>(N, K, sh_degree, campos, means, g_sh0, factors, factor_stride, A);
    else adam_sh_rank1_kernel<0><<<grid_for(N, 256), 256, smem, st>>>(N, K, sh_degree, campos, means, g_sh0, factors, factor_stride, A);
    return check_launch("adam_sh_rank1");
}

int launch_dp_sh_rank1(int K, int sh_degree, const DpRank1& A, int ctas_per_sm, cudaStream_t st) {
    if (A.n == 0 || K <= 1) return LFS_OK;
    LFS_TIMED("dp_exchange_side_sh_rank1", st);
    const size_t smem = (size_t)8 * 32 * (K - 1) * 3 * sizeof(float);
    if (smem > 200 * 1024) { set_error("dp_sh_rank1: too many SH coefficients"); return LFS_EINVAL; }
    if (smem > 48 * 1024)
        cudaFuncSetAttribute(dp_sh_rank1_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int64_t chunks = (A.lo + A.n - 1) / (32 * (K - 1) * 3) - A.lo / (32 * (K - 1) * 3) + 1;
    const int grid = grid_for(chunks * 32, 256, ctas_per_sm > 0 ? ctas_per_sm : 4);
    if (K == 16) dp_sh_rank1_kernel<16><<<grid, 256, smem, st>>>(K, sh_degree, A);
    else dp_sh_rank1_kernel<0><<<grid, 256, smem, st>>>(K, sh_degree, A);
    return check_launch("dp_sh_rank1");
}

}  // namespace lfs
