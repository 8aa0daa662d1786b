// Blend stage of the EWA (default, non --gut) rasterizer and its per-Gaussian gradient stage.
//
// Replaces blend_cu (src/training/fastgs/rasterization/include/kernels_forward.cuh:336-459), blend_backward_cu
// (include/kernels_backward.cuh:236-448), preprocess_backward_cu (:19-233) and the background blend of
// src/training/rasterization/fast_rasterizer.cpp:67.
//
// Design: a warp owns a patch of pixels and walks its tile's depth-sorted list by itself, 32 entries at a time: packed 48-byte records come to its part of
// shared memory by 16-byte asynchronous copies while the batch before is walked. It tests the 32 entries against its patch with the same
// ellipse-versus-rectangle test that built the tile lists, and walks only those that can reach it. (With the warps of a tile on one staged batch, a barrier
// apart: 1 M Gaussians, 1296x840, forward 350 us against 330, backward 617 against 546; 100 k at 256x256 142 against 89 and 200 against 125.) A thread owns
// one pixel or two horizontally adjacent ones, evaluated by the packed fp32 instructions. The backward walks the lists
// from the warp's last contributor to the front (transmittance is recovered by division, so no per-bucket state
// is stored by the forward, unlike the reference); an entry's nine gradient terms are summed over the warp by a transpose through shared memory and leave as
// one coalesced reduction of nine words.
#include "ewa.cuh"
#include "ewa_common.cuh"
#include "gsmath.cuh"
#include "pixels.cuh"
#include <math_constants.h>
#include <type_traits>

namespace lfs {
namespace {


// A warp's own staging of 32 entries, part by part, so that the lanes that test 32 entries read consecutive 16-byte words.
struct EwaStage {
    float4 r0[32], r1[32], r2[32];
    uint32_t sid[32];   // Gaussian
};
// entry `lane` of a batch of n; id: its Gaussian
__device__ __forceinline__ void stage_entries(EwaStage& st, uint32_t id, int n, const float4* __restrict__ records, int lane) {
    if (lane < n) {
        const float4* src = records + (size_t)id * 3;
        cp_async16(&st.r0[lane], src);
        cp_async16(&st.r1[lane], src + 1);
        cp_async16(&st.r2[lane], src + 2);
        st.sid[lane] = id;
    }
    cp_async_commit();
}
// which of the n staged entries can reach the 8x4 pixels from (px0, py0) on; a small margin on the threshold keeps the test conservative under rounding
__device__ __forceinline__ uint32_t cull_entries(const EwaStage& st, int n, float px0, float py0, int lane) {
    bool ok = false;
    if (lane < n) {
        const float4 r0 = st.r0[lane];
        ok = ewa_rect_contributes<true>(r0.x - 0.5f, r0.y - 0.5f, r0.z, r0.w, st.r1[lane].x, px0, px0 + 7.0f, py0, py0 + 3.0f, st.r2[lane].z + 0.01f);
    }
    return __ballot_sync(0xffffffffu, ok);
}
// The exponent of an entry at the pixels of a thread (one row). Forward and backward take the same steps, so that a pair has one alpha.
template <int PX>
__device__ __forceinline__ typename Pixels<PX>::V ewa_sigma(const float4& r0, float cyy, typename Pixels<PX>::V dx, float dy) {
    using P = Pixels<PX>;
    const typename P::V X = fma2(mul2(P::all(r0.z), dx), dx, P::all(cyy * dy * dy));
    return fma2(P::all(0.5f), X, mul2(mul2(P::all(r0.w), dx), P::all(dy)));
}
constexpr float kNegLog2e = -1.4426950408889634f;
template <int PX>
__device__ __forceinline__ typename Pixels<PX>::V chosen(const bool* which, typename Pixels<PX>::V yes, typename Pixels<PX>::V no) {
    float y[PX], n[PX];
    Pixels<PX>::get(yes, y);
    Pixels<PX>::get(no, n);
#pragma unroll
    for (int q = 0; q < PX; ++q) y[q] = which[q] ? y[q] : n[q];
    return Pixels<PX>::make(y);
}

// A warp owns a patch of 8 x 4 PX pixels and stages its own entries: no barrier, and a warp whose pixels are finished stops by itself. Which pairs count is
// decided on 8x4 pixels whatever PX is (ewa_rect_contributes says why that matters).
template <int PX>
__global__ void __launch_bounds__(128, PX == 2 ? 8 : 10) ewa_blend_fwd_kernel(
    const float4* __restrict__ records, const uint32_t* __restrict__ ids, const int32_t* __restrict__ tile_offsets,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const int32_t* __restrict__ tile_order,
    int W, int H, int tw, int n_tiles, Outsized out, float* __restrict__ image, float* __restrict__ alpha_map, int32_t* __restrict__ n_contrib) {
    using P = Pixels<PX>;
    using V = typename P::V;
    __shared__ EwaStage stages[4][2];
    EwaStage* stage = stages[threadIdx.x >> 5];
    side_by_side<PX>(out);
    const int slot = PX == 2 ? blockIdx.x : blockIdx.x >> 1;
    const int tile = tile_order ? tile_order[slot] : slot;
    if ((PX == 1 ? out.share > 0 : slot < out.slots) && is_outsized(tile_offsets[tile + 1] - tile_offsets[tile], tile_offsets[n_tiles], out) != (PX == 1)) return;
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) + (PX == 2 ? 0 : (blockIdx.x & 1) * 4);
    const int patch_j = (tile % tw) * 16 + (warp & 1) * 8, patch_i = (tile / tw) * 16 + (warp >> 1) * 4 * PX;
    const int i = patch_i + (PX == 2 ? lane >> 2 : lane >> 3), j0 = patch_j + (PX == 2 ? 2 * (lane & 3) : lane & 7);
    const bool dead = overflow && *overflow;
    const int32_t range_start = dead ? 0 : tile_offsets[tile];
    const int total = dead ? 0 : tile_offsets[tile + 1] - range_start, n_batches = (total + 31) / 32;
    const float py = (float)i + 0.5f;
    float x[PX];
    int32_t last[PX];
    bool going[PX];
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        x[q] = -((float)(j0 + q) + 0.5f);
        going[q] = i < H && j0 + q < W;
        last[q] = 0;
    }
    const V npx = P::make(x), minus_one = P::all(-1.0f);
    V T = P::all(1.0f), cr = P::all(0.f), cg = P::all(0.f), cb = P::all(0.f);
    auto batch_id = [&](int b) { return lane < total - 32 * b ? ids[range_start + 32 * b + lane] : 0u; };
    uint32_t ahead = 0;
    if (n_batches > 0) {
        stage_entries(stage[0], batch_id(0), total, records, lane);
        ahead = batch_id(1);
    }
    for (int b = 0; b < n_batches; ++b) {
        bool any_going = false;
#pragma unroll
        for (int q = 0; q < PX; ++q) any_going = any_going || going[q];
        if (!__any_sync(0xffffffffu, any_going)) break;
        if (b + 1 < n_batches) {
            // (b + 1)'s buffer was last read before the walk of b - 1 ended
            __syncwarp();
            stage_entries(stage[(b + 1) & 1], ahead, total - 32 * (b + 1), records, lane);
            ahead = batch_id(b + 2);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        const EwaStage& st = stage[b & 1];
        uint32_t bits = cull_entries(st, total - 32 * b, (float)patch_j, (float)patch_i, lane), kept = bits;
        if (PX == 2) {
            const uint32_t lower = cull_entries(st, total - 32 * b, (float)patch_j, (float)(patch_i + 4), lane);
            kept = lane < 16 ? bits : lower;
            bits |= lower;
        }
        // entries of infinite colour: zero times it is not zero, so its pixels are chosen one by one
        bool odd_colour = false;
        if (bits >> lane & 1u) odd_colour = !(fabsf(st.r1[lane].z) + fabsf(st.r1[lane].w) + fabsf(st.r2[lane].x) < CUDART_INF_F);
        uint32_t odd = __ballot_sync(0xffffffffu, odd_colour);
        uint32_t mine[PX];   // the entries that a pixel still asks
#pragma unroll
        for (int q = 0; q < PX; ++q) mine[q] = going[q] ? kept : 0u;
        auto blend = [&](int t, uint32_t lowest, auto finite) {
            const float4 r0 = st.r0[t], r1 = st.r1[t];
            const V dx = add2(P::all(r0.x), npx), sigma = ewa_sigma<PX>(r0, r1.x, dx, r0.y - py);
            float s[PX], e[PX], a[PX];
            P::get(sigma, s);
            P::get(mul2(sigma, P::all(kNegLog2e)), e);
#pragma unroll
            for (int q = 0; q < PX; ++q) e[q] = exp2_approx(e[q]);
            P::get(mul2(P::all(r1.y), P::make(e)), a);
            bool valid[PX];
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                a[q] = fminf(a[q], kEwaMaxAlpha);
                valid[q] = (mine[q] & lowest) != 0u && !(s[q] < 0.0f) && !(a[q] < kEwaMinAlpha);
                if (!valid[q]) a[q] = 0.f;
            }
            V al = P::make(a);
            V next_T = mul2(T, mul2(add2(al, minus_one), minus_one));
            float nt[PX];
            P::get(next_T, nt);
            bool stops = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) stops = stops || nt[q] < kEwaMinTransmittance;   // no pixel without alpha comes here: its T is not below
            if (stops) {
                float t0[PX];
                P::get(T, t0);
#pragma unroll
                for (int q = 0; q < PX; ++q)
                    if (nt[q] < kEwaMinTransmittance) { valid[q] = going[q] = false; mine[q] = 0u; a[q] = 0.f; nt[q] = t0[q]; }
                al = P::make(a);
                next_T = P::make(nt);
            }
            const V w = mul2(T, al);
            const V red = fma2(w, P::all(r1.z), cr), green = fma2(w, P::all(r1.w), cg), blue = fma2(w, P::all(st.r2[t].x), cb);
            if constexpr (decltype(finite)::value) {
                cr = red; cg = green; cb = blue;
            } else {
                cr = chosen<PX>(valid, red, cr); cg = chosen<PX>(valid, green, cg); cb = chosen<PX>(valid, blue, cb);
            }
            T = next_T;
#pragma unroll
            for (int q = 0; q < PX; ++q) last[q] = valid[q] ? 32 * b + t + 1 : last[q];
        };
        while (bits) {
            // up to the next odd one, or all
            uint32_t run = bits & ((odd & (0u - odd)) - 1u);
            bits &= ~run;
            while (run) {
                const uint32_t lowest = run & (0u - run);
                blend(__ffs(run) - 1, lowest, std::true_type{});
                run &= run - 1;
            }
            if (odd) {
                const uint32_t lowest = odd & (0u - odd);
                blend(__ffs(odd) - 1, lowest, std::false_type{});
                odd &= odd - 1;
                bits &= ~lowest;
            }
        }
    }
    cp_async_wait<0>();
    float Tq[PX], rq[PX], gq[PX], bq[PX];
    P::get(T, Tq); P::get(cr, rq); P::get(cg, gq); P::get(cb, bq);
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        if (!(i < H && j0 + q < W)) continue;
        const size_t pid = (size_t)i * W + j0 + q, np = (size_t)W * H;
        if (background) { rq[q] += Tq[q] * background[0]; gq[q] += Tq[q] * background[1]; bq[q] += Tq[q] * background[2]; }
        image[pid] = rq[q];
        image[np + pid] = gq[q];
        image[2 * np + pid] = bq[q];
        alpha_map[pid] = 1.0f - Tq[q];
        n_contrib[pid] = last[q];
    }
}

// 9 values per lane -> per-value sums over the warp, value k left in lanes 2k and 2k+1 (lanes 18..31 repeat value 8), through shared memory owned by the
// warp: row k (36 floats, 32 used) holds value k of the 32 lanes. The row stride of 36 floats puts the 16-byte loads of one quarter-warp (lane = 2 k + h
// reads the 16 lanes of half h of row k) on eight different bank groups, and the scalar stores of one row are contiguous. The rows are written when an
// entry has been evaluated and summed in the shadow of the next one's evaluation; the closing shuffle needs every lane's sum, hence every lane's loads,
// before any lane writes the rows again.
constexpr int kRedStride = 36, kEwaSums = 9;
struct EwaBwdWarp {
    EwaStage stage[2];
    float red[kEwaSums * kRedStride];
};

template <int PX>
__global__ void __launch_bounds__(128, PX == 2 ? 6 : 8) ewa_blend_bwd_kernel(
    const float4* __restrict__ records, const uint32_t* __restrict__ ids, const int32_t* __restrict__ tile_offsets,
    const int32_t* __restrict__ overflow, const float* __restrict__ background, const int32_t* __restrict__ tile_order,
    int W, int H, int tw, int n_tiles, Outsized out, const float* __restrict__ alpha_map, const int32_t* __restrict__ n_contrib,
    const float* __restrict__ grad_image,
    const float* __restrict__ grad_alpha, float* __restrict__ accum) {
    using P = Pixels<PX>;
    using V = typename P::V;
    __shared__ EwaBwdWarp warps[4];
    EwaBwdWarp& sm = warps[threadIdx.x >> 5];
    side_by_side<PX>(out);
    if (overflow && *overflow) return;
    const int slot = PX == 2 ? blockIdx.x : blockIdx.x >> 1;
    const int tile = tile_order ? tile_order[slot] : slot;
    if ((PX == 1 ? out.share > 0 : slot < out.slots) && is_outsized(tile_offsets[tile + 1] - tile_offsets[tile], tile_offsets[n_tiles], out) != (PX == 1)) return;
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) + (PX == 2 ? 0 : (blockIdx.x & 1) * 4);
    // warps tile the 16x16 block as patches of 8 x 4 PX pixels: one or two of the forward's 8x4 patches, one above the other
    const int patch_j = (tile % tw) * 16 + (warp & 1) * 8, patch_i = (tile / tw) * 16 + (warp >> 1) * 4 * PX;
    const int i = patch_i + (PX == 2 ? lane >> 2 : lane >> 3), j0 = patch_j + (PX == 2 ? 2 * (lane & 3) : lane & 7);
    const float py = (float)i + 0.5f;
    const size_t np = (size_t)W * H;
    const int32_t range_start = tile_offsets[tile];

    float x[PX], r[PX], g[PX], bl[PX], tf[PX], bh[PX];
    int32_t my_last[PX];   // entries at list positions < my_last can contribute
    int32_t total = 0;
#pragma unroll
    for (int q = 0; q < PX; ++q) {
        const int j = j0 + q;
        const bool inside = i < H && j < W;
        const size_t pid = inside ? (size_t)i * W + j : 0;
        x[q] = -((float)j + 0.5f);
        r[q] = inside ? grad_image[pid] : 0.f; g[q] = inside ? grad_image[np + pid] : 0.f; bl[q] = inside ? grad_image[2 * np + pid] : 0.f;
        tf[q] = inside ? 1.0f - alpha_map[pid] : 1.0f;
        float ga = (inside && grad_alpha) ? grad_alpha[pid] : 0.f;
        if (background) ga -= r[q] * background[0] + g[q] * background[1] + bl[q] * background[2];  // image = blend + (1 - alpha) bg
        bh[q] = ga * tf[q];
        my_last[q] = inside ? n_contrib[pid] : 0;
        total = max(total, my_last[q]);
    }
    const V npx = P::make(x), gr = P::make(r), gg = P::make(g), gb = P::make(bl), minus_one = P::all(-1.0f), one = P::all(1.0f);
    V T = P::make(tf);
    V behind = P::make(bh);   // (colour . gradient) already blended behind the entry being walked, minus the share of alpha's gradient
    // the warp walks from its own deepest contributor to the front
    total = __reduce_max_sync(0xffffffffu, total);
    if (total <= 0) return;
    const int n_batches = (total + 31) / 32;
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t pending = kNone;   // Gaussian whose sums lie in `red`
    const ulonglong2* red_half = reinterpret_cast<const ulonglong2*>(sm.red + min(lane >> 1, kEwaSums - 1) * kRedStride + 16 * (lane & 1));
    const bool red_lane = (lane & 1) == 0 && lane < 2 * kEwaSums;
    auto flush = [&](uint32_t id) {
        const ulonglong2 x0 = red_half[0], x1 = red_half[1], x2 = red_half[2], x3 = red_half[3];
        float sum = Pixels<2>::sum(add2(add2(add2(x0.x, x0.y), add2(x1.x, x1.y)), add2(add2(x2.x, x2.y), add2(x3.x, x3.y))));
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (red_lane && id != kNone) atomicAdd(accum + (size_t)id * 12 + (lane >> 1), sum);
    };
    auto batch_id = [&](int b) { return lane < total - 32 * b ? ids[range_start + total - 1 - 32 * b - lane] : 0u; };
    stage_entries(sm.stage[0], batch_id(0), total, records, lane);
    uint32_t ahead = batch_id(1);
    for (int b = 0; b < n_batches; ++b) {
        const int32_t batch_top = total - 1 - 32 * b;   // slot t holds the tile's list position batch_top - t
        if (b + 1 < n_batches) {
            __syncwarp();
            stage_entries(sm.stage[(b + 1) & 1], ahead, total - 32 * (b + 1), records, lane);
            ahead = batch_id(b + 2);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncwarp();
        const EwaStage& st = sm.stage[b & 1];
        // The ellipse-versus-rectangle test misses a rectangle now and then (ewa_rect_contributes says when), and differently for
        // rectangles of another shape, so a pair counts only if the forward's own 8x4 patch kept it: a pixel that the forward skipped
        // must not enter the transmittance here.
        uint32_t bits = cull_entries(st, total - 32 * b, (float)patch_j, (float)patch_i, lane), mine = bits;
        if (PX == 2) {
            const uint32_t lower = cull_entries(st, total - 32 * b, (float)patch_j, (float)(patch_i + 4), lane);
            mine = lane < 16 ? bits : lower;
            bits |= lower;
        }
        while (bits) {
            const int t = __ffs(bits) - 1;
            const bool kept = PX == 1 || (mine & bits & (0u - bits)) != 0u;
            bits &= bits - 1;
            const float4 r0 = st.r0[t], r1 = st.r1[t];
            const float blue = st.r2[t].x, dy = r0.y - py;
            flush(pending);
            pending = kNone;
            const V dx = add2(P::all(r0.x), npx), sigma = ewa_sigma<PX>(r0, r1.x, dx, dy);
            float s[PX], e[PX], a[PX];
            P::get(sigma, s);
            P::get(mul2(sigma, P::all(kNegLog2e)), e);
#pragma unroll
            for (int q = 0; q < PX; ++q) e[q] = exp2_approx(e[q]);
            P::get(mul2(P::all(r1.y), P::make(e)), a);
            bool any_valid = false;
#pragma unroll
            for (int q = 0; q < PX; ++q) {
                a[q] = fminf(a[q], kEwaMaxAlpha);
                const bool valid = kept && batch_top - t < my_last[q] && !(s[q] < 0.0f) && !(a[q] < kEwaMinAlpha);
                any_valid = any_valid || valid;
                if (!valid) a[q] = 0.f;  // every term below is then exactly zero for this pixel
            }
            if (!__any_sync(0xffffffffu, any_valid)) continue;
            const V al = P::make(a), na = add2(al, minus_one);
            float y0[PX];
            P::get(na, y0);
#pragma unroll
            for (int q = 0; q < PX; ++q) y0[q] = rcp_approx(-y0[q]);
            // 1 / (1 - a), 1 - a in [0.001, 1]: the hardware estimate and one Newton step (relative error below 2^-23)
            const V y = P::make(y0), rcp = fma2(y, fma2(na, y, one), y);
            T = mul2(T, rcp);  // transmittance in front of this entry
            const V wgt = mul2(T, al);
            // colour . gradient of this entry: the colours only ever meet the output gradient in this product
            const V cv = fma2(P::all(r1.z), gr, fma2(P::all(r1.w), gg, mul2(P::all(blue), gb)));
            const V dL_da = fma2(cv, T, mul2(rcp, behind));
            behind = fma2(mul2(cv, minus_one), wgt, behind);
            const V adl = mul2(al, dL_da);
            const V hx = mul2(adl, dx), hy = mul2(adl, P::all(dy));    // minus the gradient of the exponent, times the offset
            // sums of a dL/da times (1, dx, dy, dx^2, dx dy, dy^2): the conic multiplies them after the reduction
            const float hys = P::sum(hy);
            auto put = [&](int k, float v) { sm.red[k * kRedStride + lane] = v; };
            put(0, P::sum(hx)); put(1, hys); put(2, P::sum(mul2(hx, dx))); put(3, P::sum(hx) * dy); put(4, hys * dy); put(5, P::sum(adl));
            put(6, P::sum(mul2(wgt, gr))); put(7, P::sum(mul2(wgt, gg))); put(8, P::sum(mul2(wgt, gb)));
            pending = st.sid[t];
            __syncwarp();
        }
    }
    flush(pending);
}

// ---------------------------------------------------------------------------------------------
// Per-Gaussian gradient stage: from (d mean2d, d conic, sum alpha dL/dalpha, d colour) to the six raw tensors.
// cov2d = A Sigma A^T + 0.3 I with A = J W (2x3), Sigma = R diag(exp(2 s)) R^T, conic = cov2d^-1.
// ---------------------------------------------------------------------------------------------
// Each warp handles 32 consecutive Gaussians per iteration: their shN rows ((K-1)*3 floats each, contiguous in
// memory) are read as one coalesced run into shared memory, every lane then works on its own row in place
// (coefficient in, gradient out), and the 32 gradient rows leave as one coalesced run.
// capped at 64 registers (the compiler takes 114 unasked): this stage is latency bound and wants the fourth resident CTA
// W2C: also the camera-pose gradient of kernels_backward.cuh:160-173, sum over the Gaussians that reached a tile of
// (gradient of the camera-space mean) x (mean, 1), rows 0..2 of a [4,4] matrix: per warp a shuffle reduction, per CTA 12
// shared sums, 12 atomics per CTA at the end. A separate instantiation, so the default one keeps its registers.
template <bool W2C>
__global__ void __launch_bounds__(256, 4) ewa_epilogue_kernel(
    int N, int K, const float* __restrict__ means, const float* __restrict__ shN, const float* __restrict__ scaling_raw,
    const float* __restrict__ rotation_raw, EwaCamera cam, const int32_t* __restrict__ n_touched, const float4* __restrict__ records,
    const float* __restrict__ accum, float* __restrict__ g_means, float* __restrict__ g_sh0, float* __restrict__ g_shN,
    float* __restrict__ g_scaling, float* __restrict__ g_rotation, float* __restrict__ g_opacity, int accumulate,
    float* __restrict__ densification_info, float* __restrict__ grad_w2c) {
    extern __shared__ __align__(16) float s_rows[];
    __shared__ float s_pose[8][12];
    const bool rows_aligned = (reinterpret_cast<uintptr_t>(shN) & 15) == 0;
    const bool out_aligned = (reinterpret_cast<uintptr_t>(g_shN) & 15) == 0;
    if (W2C) {
        if (threadIdx.x < 96) s_pose[threadIdx.x / 12][threadIdx.x % 12] = 0.f;
        __syncthreads();
    }
    float r1[4], r2[4], r3[4], campos[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) { r1[k] = cam.w2c[k]; r2[k] = cam.w2c[4 + k]; r3[k] = cam.w2c[8 + k]; }
#pragma unroll
    for (int k = 0; k < 3; ++k) campos[k] = cam.campos[k];
    const int rest = (K - 1) * 3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* my = s_rows + (size_t)warp * 32 * rest;
    const int n_chunks = (N + 31) / 32;
    const int warps_total = gridDim.x * (blockDim.x >> 5);
    const int nb = cam.active_sh_bases > 9 ? 16 : cam.active_sh_bases > 4 ? 9 : cam.active_sh_bases > 1 ? 4 : 1;
    for (int chunk = blockIdx.x * (blockDim.x >> 5) + warp; chunk < n_chunks; chunk += warps_total) {
        const int i = chunk * 32 + lane;
        const bool in_range = i < N;
        const bool visible = in_range && n_touched[i] > 0;
        const bool any_visible = __any_sync(0xffffffffu, visible);
        const int n_rows = min(32, N - chunk * 32);
        const int total = n_rows * rest;
        float* dst_rows = g_shN + (size_t)chunk * 32 * rest;
        if (!any_visible) {
            // nothing in this chunk reached a tile: zeros (or untouched when accumulating)
            if (!accumulate) {
                if (g_shN) for (int k = lane; k < total; k += 32) dst_rows[k] = 0.f;
                if (in_range) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) { g_means[i * 3 + k] = 0.f; g_sh0[i * 3 + k] = 0.f; g_scaling[i * 3 + k] = 0.f; }
                    reinterpret_cast<float4*>(g_rotation)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    g_opacity[i] = 0.f;
                }
            }
            continue;
        }
        if (nb > 1) {
            // 16-byte asynchronous copies where the tensor allows it (a chunk starts at a multiple of 32 rows): one round trip
            // for the chunk instead of one per register batch
            const float* src_rows = shN + (size_t)chunk * 32 * rest;
            const int total4 = rows_aligned ? total >> 2 : 0;
            for (int k = lane; k < total4; k += 32) cp_async16(my + k * 4, src_rows + k * 4);
            cp_async_commit();
            for (int k = total4 * 4 + lane; k < total; k += 32) my[k] = src_rows[k];
            cp_async_wait<0>();
        }
        __syncwarp();
        float* out_rest = my + lane * rest;   // this lane's row: coefficients now, gradients afterwards
        float gm[3] = {0.f, 0.f, 0.f}, gs[3] = {0.f, 0.f, 0.f}, gq[4] = {0.f, 0.f, 0.f, 0.f}, g0[3] = {0.f, 0.f, 0.f}, go = 0.f;
        float pose[12];
        if (W2C) {
#pragma unroll
            for (int k = 0; k < 12; ++k) pose[k] = 0.f;
        }
        if (!visible) {
            for (int k = 0; k < rest; ++k) out_rest[k] = 0.f;
        } else {
        float acc[12];
        const float4* a4 = reinterpret_cast<const float4*>(accum) + (size_t)i * 3;
#pragma unroll
        for (int k = 0; k < 3; ++k) { const float4 t = a4[k]; acc[k * 4] = t.x; acc[k * 4 + 1] = t.y; acc[k * 4 + 2] = t.z; acc[k * 4 + 3] = t.w; }
        const float4 rc0 = records[(size_t)i * 3], rc1 = records[(size_t)i * 3 + 1], rc2 = records[(size_t)i * 3 + 2];
        {
            // the blend stage sums a dL/da (dx, dy | dx^2, dx dy, dy^2); d exponent / d mean2d = -conic (dx, dy),
            // d exponent / d conic = -(dx^2, dx dy, dy^2) / 2 (symmetric-entry convention)
            const float sx = acc[0], sy = acc[1];
            acc[0] = -(rc0.z * sx + rc0.w * sy);
            acc[1] = -(rc0.w * sx + rc1.x * sy);
            acc[2] *= -0.5f; acc[3] *= -0.5f; acc[4] *= -0.5f;
        }
        const uint32_t mask = __float_as_uint(rc2.y);
        const float gc[3] = {(mask & 1u) ? acc[6] : 0.f, (mask & 2u) ? acc[7] : 0.f, (mask & 4u) ? acc[8] : 0.f};
        go = acc[5] * (1.0f - rc1.y);
        const float m0 = means[i * 3], m1 = means[i * 3 + 1], m2 = means[i * 3 + 2];
        // ---- colour: SH coefficients and, through the view direction, the mean
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) g0[ch] = 0.28209479177387814f * gc[ch];
        float dmc[3] = {0.f, 0.f, 0.f};
        if (nb > 1) {
            const float xr = m0 - campos[0], yr = m1 - campos[1], zr = m2 - campos[2];
            const float inv = rsqrtf(xr * xr + yr * yr + zr * zr);
            const float x = xr * inv, y = yr * inv, z = zr * inv;
            const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, xz = x * z, yz = y * z;
            const float* co = out_rest;
            float gd[3] = {0.f, 0.f, 0.f};
            // basis value B and its derivative (Dx, Dy, Dz) with respect to the unit direction, one row at a time
            auto row = [&](int k, float B, float Dx, float Dy, float Dz) {
                const float c0 = co[(k - 1) * 3], c1 = co[(k - 1) * 3 + 1], c2 = co[(k - 1) * 3 + 2];
                const float cgd = c0 * gc[0] + c1 * gc[1] + c2 * gc[2];
                gd[0] += Dx * cgd; gd[1] += Dy * cgd; gd[2] += Dz * cgd;
                out_rest[(k - 1) * 3] = B * gc[0]; out_rest[(k - 1) * 3 + 1] = B * gc[1]; out_rest[(k - 1) * 3 + 2] = B * gc[2];
            };
            row(1, -0.48860251190291987f * y, 0.f, -0.48860251190291987f, 0.f);
            row(2, 0.48860251190291987f * z, 0.f, 0.f, 0.48860251190291987f);
            row(3, -0.48860251190291987f * x, -0.48860251190291987f, 0.f, 0.f);
            if (nb > 4) {
                row(4, 1.0925484305920792f * xy, 1.0925484305920792f * y, 1.0925484305920792f * x, 0.f);
                row(5, -1.0925484305920792f * yz, 0.f, -1.0925484305920792f * z, -1.0925484305920792f * y);
                row(6, 0.94617469575755997f * zz - 0.31539156525251999f, 0.f, 0.f, 1.8923493915151202f * z);
                row(7, -1.0925484305920792f * xz, -1.0925484305920792f * z, 0.f, -1.0925484305920792f * x);
                row(8, 0.54627421529603959f * xx - 0.54627421529603959f * yy, 1.0925484305920792f * x, -1.0925484305920792f * y, 0.f);
            }
            if (nb > 9) {
                row(9, 0.59004358992664352f * y * (-3.0f * xx + yy), -3.5402615395598609f * xy, -1.7701307697799304f * xx + 1.7701307697799304f * yy, 0.f);
                row(10, 2.8906114426405538f * xy * z, 2.8906114426405538f * yz, 2.8906114426405538f * xz, 2.8906114426405538f * xy);
                row(11, 0.45704579946446572f * y * (1.0f - 5.0f * zz), 0.f, 0.45704579946446572f - 2.2852289973223288f * zz, -4.5704579946446566f * yz);
                row(12, 0.3731763325901154f * z * (5.0f * zz - 3.0f), 0.f, 0.f, 5.597644988851731f * zz - 1.1195289977703462f);
                row(13, 0.45704579946446572f * x * (1.0f - 5.0f * zz), 0.45704579946446572f - 2.2852289973223288f * zz, 0.f, -4.5704579946446566f * xz);
                row(14, 1.4453057213202769f * z * (xx - yy), 2.8906114426405538f * xz, -2.8906114426405538f * yz, 1.4453057213202769f * xx - 1.4453057213202769f * yy);
                row(15, 0.59004358992664352f * x * (-xx + 3.0f * yy), -1.7701307697799304f * xx + 1.7701307697799304f * yy, 3.5402615395598609f * xy, 0.f);
            }
            for (int k = (nb - 1) * 3; k < rest; ++k) out_rest[k] = 0.f;
            // through the normalisation: (|r|^2 I - r r^T) gd / |r|^3
            const float xxr = xr * xr, yyr = yr * yr, zzr = zr * zr, xyr = xr * yr, xzr = xr * zr, yzr = yr * zr;
            const float n2 = xxr + yyr + zzr;
            const float s = rsqrtf(n2 * n2 * n2);
            dmc[0] = ((yyr + zzr) * gd[0] - xyr * gd[1] - xzr * gd[2]) * s;
            dmc[1] = (-xyr * gd[0] + (xxr + zzr) * gd[1] - yzr * gd[2]) * s;
            dmc[2] = (-xzr * gd[0] - yzr * gd[1] + (xxr + yyr) * gd[2]) * s;
        } else {
            for (int k = 0; k < rest; ++k) out_rest[k] = 0.f;
        }
        // ---- geometry, recomputed as in the forward
        const float depth = r3[0] * m0 + r3[1] * m1 + r3[2] * m2 + r3[3];
        const float x = (r1[0] * m0 + r1[1] * m1 + r1[2] * m2 + r1[3]) / depth;
        const float y = (r2[0] * m0 + r2[1] * m1 + r2[2] * m2 + r2[3]) / depth;
        const float var[3] = {expf(2.0f * scaling_raw[i * 3]), expf(2.0f * scaling_raw[i * 3 + 1]), expf(2.0f * scaling_raw[i * 3 + 2])};
        const float4 q = reinterpret_cast<const float4*>(rotation_raw)[i];
        const float qr = q.x, qx = q.y, qy = q.z, qz = q.w;
        const float n = qr * qr + qx * qx + qy * qy + qz * qz;
        const float pxx = 2.0f * qx * qx / n, pyy = 2.0f * qy * qy / n, pzz = 2.0f * qz * qz / n;
        const float pxy = 2.0f * qx * qy / n, pxz = 2.0f * qx * qz / n, pyz = 2.0f * qy * qz / n;
        const float prx = 2.0f * qr * qx / n, pry = 2.0f * qr * qy / n, prz = 2.0f * qr * qz / n;
        const float R[9] = {1.0f - (pyy + pzz), pxy - prz, pry + pxz, prz + pxy, 1.0f - (pxx + pzz), pyz - prx, pxz - pry, prx + pyz, 1.0f - (pxx + pyy)};
        float RS[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k) RS[r * 3 + k] = R[r * 3 + k] * var[k];
        auto rowdot = [&](int a, int b) { return RS[a * 3] * R[b * 3] + RS[a * 3 + 1] * R[b * 3 + 1] + RS[a * 3 + 2] * R[b * 3 + 2]; };
        const float Sg[6] = {rowdot(0, 0), rowdot(0, 1), rowdot(0, 2), rowdot(1, 1), rowdot(1, 2), rowdot(2, 2)};
        const float Wf = (float)cam.W, Hf = (float)cam.H;
        const float tx = fminf(fmaxf(x, (-0.15f * Wf - cam.cx) / cam.fx), (1.15f * Wf - cam.cx) / cam.fx);
        const float ty = fminf(fmaxf(y, (-0.15f * Hf - cam.cy) / cam.fy), (1.15f * Hf - cam.cy) / cam.fy);
        const float j11 = cam.fx / depth, j13 = -j11 * tx, j22 = cam.fy / depth, j23 = -j22 * ty;
        float A1[3], A2[3], B1[3], B2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) { A1[k] = j11 * r1[k] + j13 * r3[k]; A2[k] = j22 * r2[k] + j23 * r3[k]; }
        B1[0] = A1[0] * Sg[0] + A1[1] * Sg[1] + A1[2] * Sg[2];
        B1[1] = A1[0] * Sg[1] + A1[1] * Sg[3] + A1[2] * Sg[4];
        B1[2] = A1[0] * Sg[2] + A1[1] * Sg[4] + A1[2] * Sg[5];
        B2[0] = A2[0] * Sg[0] + A2[1] * Sg[1] + A2[2] * Sg[2];
        B2[1] = A2[0] * Sg[1] + A2[1] * Sg[3] + A2[2] * Sg[4];
        B2[2] = A2[0] * Sg[2] + A2[1] * Sg[4] + A2[2] * Sg[5];
        const float a = (B1[0] * A1[0] + B1[1] * A1[1] + B1[2] * A1[2]) + kEwaDilation;
        const float b = B1[0] * A2[0] + B1[1] * A2[1] + B1[2] * A2[2];
        const float c = (B2[0] * A2[0] + B2[1] * A2[1] + B2[2] * A2[2]) + kEwaDilation;
        const float rcp = 1.0f / (a * c - b * b), rcp2 = rcp * rcp;
        // gradient of conic = cov2d^-1 (symmetric-entry convention: the off-diagonal sum was accumulated with 1/2)
        const float kx = acc[2], ky = acc[3], kz = acc[4];
        const float hx = rcp2 * (2.0f * (b * c) * ky - (c * c) * kx - (b * b) * kz);
        const float hy = rcp2 * ((b * c) * kx - ((a * c) + (b * b)) * ky + (a * b) * kz);
        const float hz = rcp2 * (2.0f * (a * b) * ky - (b * b) * kx - (a * a) * kz);
        // d/d Sigma = A^T H A
        float S[6];
        S[0] = (A1[0] * A1[0]) * hx + 2.0f * (A1[0] * A2[0]) * hy + (A2[0] * A2[0]) * hz;
        S[1] = (A1[0] * A1[1]) * hx + (A1[0] * A2[1] + A1[1] * A2[0]) * hy + (A2[0] * A2[1]) * hz;
        S[2] = (A1[0] * A1[2]) * hx + (A1[0] * A2[2] + A1[2] * A2[0]) * hy + (A2[0] * A2[2]) * hz;
        S[3] = (A1[1] * A1[1]) * hx + 2.0f * (A1[1] * A2[1]) * hy + (A2[1] * A2[1]) * hz;
        S[4] = (A1[1] * A1[2]) * hx + (A1[1] * A2[2] + A1[2] * A2[1]) * hy + (A2[1] * A2[2]) * hz;
        S[5] = (A1[2] * A1[2]) * hx + 2.0f * (A1[2] * A2[2]) * hy + (A2[2] * A2[2]) * hz;
        // d/d A = 2 H (A Sigma), then the four non-constant entries of J
        float dA1[3], dA2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) { dA1[k] = 2.0f * (B1[k] * hx + B2[k] * hy); dA2[k] = 2.0f * (B1[k] * hy + B2[k] * hz); }
        const float dj11 = r1[0] * dA1[0] + r1[1] * dA1[1] + r1[2] * dA1[2];
        const float dj22 = r2[0] * dA2[0] + r2[1] * dA2[1] + r2[2] * dA2[2];
        const float dj13 = r3[0] * dA1[0] + r3[1] * dA1[1] + r3[2] * dA1[2];
        const float dj23 = r3[0] * dA2[0] + r3[1] * dA2[1] + r3[2] * dA2[2];
        const float m2x = acc[0], m2y = acc[1];
        const float dcx = j11 * (m2x - dj13 / depth), dcy = j22 * (m2y - dj23 / depth);
        const float dcz = -j11 * (x * m2x + (dj11 - 2.0f * tx * dj13) / depth) - j22 * (y * m2y + (dj22 - 2.0f * ty * dj23) / depth);
#pragma unroll
        for (int k = 0; k < 3; ++k) gm[k] = (r1[k] * dcx + r2[k] * dcy + r3[k] * dcz) + dmc[k];
        if (W2C) {
            const float dc[3] = {dcx, dcy, dcz}, mh[4] = {m0, m1, m2, 1.0f};
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) pose[r * 4 + k] = dc[r] * mh[k];
        }
        // variances (columns of R) and the log-scale chain
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float u = R[k], v = R[3 + k], w = R[6 + k];
            gs[k] = 2.0f * var[k] * (u * u * S[0] + v * v * S[3] + w * w * S[5] + 2.0f * (u * v * S[1] + u * w * S[2] + v * w * S[4]));
        }
        // rotation: d/dR = 2 S (R diag(var)), R is linear in the products p_ab = 2 q_a q_b / |q|^2
        const float Sm[9] = {S[0], S[1], S[2], S[1], S[3], S[4], S[2], S[4], S[5]};
        float dR[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k) dR[r * 3 + k] = 2.0f * (RS[k] * Sm[r * 3] + RS[3 + k] * Sm[r * 3 + 1] + RS[6 + k] * Sm[r * 3 + 2]);
        const float dxx = -dR[4] - dR[8], dyy = -dR[0] - dR[8], dzz = -dR[0] - dR[4];
        const float dxy = dR[1] + dR[3], dxz = dR[2] + dR[6], dyz = dR[5] + dR[7];
        const float drx = dR[7] - dR[5], dry = dR[2] - dR[6], drz = dR[3] - dR[1];
        const float nh = pxx * dxx + pyy * dyy + pzz * dzz + pxy * dxy + pxz * dxz + pyz * dyz + prx * drx + pry * dry + prz * drz;
        gq[0] = 2.0f * (qx * drx + qy * dry + qz * drz - qr * nh) / n;
        gq[1] = 2.0f * (2.0f * qx * dxx + qy * dxy + qz * dxz + qr * drx - qx * nh) / n;
        gq[2] = 2.0f * (2.0f * qy * dyy + qx * dxy + qz * dyz + qr * dry - qy * nh) / n;
        gq[3] = 2.0f * (2.0f * qz * dzz + qx * dxz + qy * dyz + qr * drz - qz * nh) / n;
        if (densification_info) {
            densification_info[i] += 1.0f;
            const float sx = m2x * (0.5f * Wf), sy = m2y * (0.5f * Hf);
            densification_info[N + i] += sqrtf(sx * sx + sy * sy);
        }
        }  // visible
        __syncwarp();
        if (W2C) {
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                float v = pose[k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) s_pose[warp][k] += v;
            }
        }
        if (!g_shN) {
            // the caller rebuilds these rows from the sh0 gradient (lfs_ewa_adam_step_rank1_sh)
        } else {
            store_rows(dst_rows, my, total, lane, out_aligned, accumulate != 0);
        }
        __syncwarp();
        if (in_range && (visible || !accumulate)) {
            if (accumulate) {
#pragma unroll
                for (int k = 0; k < 3; ++k) { g_means[i * 3 + k] += gm[k]; g_sh0[i * 3 + k] += g0[k]; g_scaling[i * 3 + k] += gs[k]; }
#pragma unroll
                for (int k = 0; k < 4; ++k) g_rotation[i * 4 + k] += gq[k];
                g_opacity[i] += go;
            } else {
#pragma unroll
                for (int k = 0; k < 3; ++k) { g_means[i * 3 + k] = gm[k]; g_sh0[i * 3 + k] = g0[k]; g_scaling[i * 3 + k] = gs[k]; }
                reinterpret_cast<float4*>(g_rotation)[i] = make_float4(gq[0], gq[1], gq[2], gq[3]);
                g_opacity[i] = go;
            }
        }
    }
    if (W2C) {
        __syncthreads();
        if (threadIdx.x < 12) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) v += s_pose[w][threadIdx.x];
            if (v != 0.f) atomicAdd(grad_w2c + threadIdx.x, v);
        }
    }
}

}  // namespace

int launch_ewa_blend_fwd(const EwaBlendArgs& a, float* image, float* alpha, int32_t* n_contrib, cudaStream_t st) {
    const int n_tiles = a.tw * a.th;
    if (n_tiles == 0) return LFS_OK;
    LFS_TIMED("ewa_blend_fwd", st);
    const Outsized out = outsized_lists(a.tile_order, n_tiles);   // the forward always leaves a launch order
#define LFS_EWA_FWD(LAUNCH, PX, TILES, OUT)                                                                                         \
    LAUNCH(ewa_blend_fwd_kernel<PX>, (TILES) * (2 / PX), 128, 0, st, a.records, a.instance_ids, a.tile_offsets, a.overflow, a.background,  \
                                                                 a.tile_order, a.W, a.H, a.tw, n_tiles, OUT, image, alpha, n_contrib)
    // Two pixels per thread where the patches of twice the size still fill the GPU. us with one and two, 100 k Gaussians: 920 tiles 81 and 95, 2,170 tiles 125
    // and 121 (400 k: 160 and 166), 4,293 tiles 201 and 183.
    if (n_tiles >= 16 * num_sms()) { LFS_EWA_FWD(launch, 1, out.slots, out); LFS_EWA_FWD(launch_beside, 2, n_tiles, out); }
    else LFS_EWA_FWD(launch, 1, n_tiles, Outsized{});
#undef LFS_EWA_FWD
    return check_launch("ewa_blend_fwd");
}

int launch_ewa_blend_bwd(const EwaBlendArgs& a, const float* alpha, const int32_t* n_contrib, const float* grad_image,
                         const float* grad_alpha, float* accum, cudaStream_t st) {
    const int n_tiles = a.tw * a.th;
    if (n_tiles == 0) return LFS_OK;
    LFS_TIMED("ewa_blend_bwd", st);
    const Outsized out = outsized_lists(a.tile_order, n_tiles);
#define LFS_EWA_BWD(LAUNCH, PX, TILES, OUT)                                                                                         \
    LAUNCH(ewa_blend_bwd_kernel<PX>, (TILES) * (2 / PX), 128, 0, st, a.records, a.instance_ids, a.tile_offsets, a.overflow, a.background,      \
                                                           a.tile_order, a.W, a.H, a.tw, n_tiles, OUT, alpha, n_contrib, grad_image, grad_alpha,   \
                                                           accum)
    // Two pixels per thread as in the forward; the sums of an entry are then formed half as often. us with one and two, 100 k Gaussians: 256 tiles 125 and 205, 510
    // tiles 134 and 147, 920 tiles 164 and 144, 4,293 tiles 473 and 310.
    if (n_tiles >= 4 * num_sms()) { LFS_EWA_BWD(launch, 1, out.slots, out); LFS_EWA_BWD(launch_beside, 2, n_tiles, out); }
    else LFS_EWA_BWD(launch, 1, n_tiles, Outsized{});
#undef LFS_EWA_BWD
    return check_launch("ewa_blend_bwd");
}

int launch_ewa_epilogue(int N, int K, const lfs_splats& p, const EwaCamera& cam, const int32_t* n_touched, const float4* records,
                        const float* accum, const lfs_splats& g, int accumulate, float* densification_info, float* grad_w2c,
                        cudaStream_t st) {
    if (grad_w2c && !accumulate) cudaMemsetAsync(grad_w2c, 0, 16 * sizeof(float), st);
    if (N == 0) return LFS_OK;
    LFS_TIMED("ewa_epilogue", st);
    const size_t smem = (size_t)8 * 32 * (K - 1) * 3 * sizeof(float);
    if (smem > 200 * 1024) { set_error("ewa_epilogue: too many SH coefficients"); return LFS_EINVAL; }
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(ewa_epilogue_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(ewa_epilogue_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
#define LFS_EWA_EPILOGUE(W2C)                                                                                                       \
    ewa_epilogue_kernel<W2C><<<grid_for(N, 256), 256, smem, st>>>(N, K, p.means, p.shN, p.scaling_raw, p.rotation_raw, cam, n_touched, \
                                                                 records, accum, g.means, g.sh0, g.shN, g.scaling_raw, g.rotation_raw, \
                                                                 g.opacity_raw, accumulate, densification_info, grad_w2c)
    if (grad_w2c) LFS_EWA_EPILOGUE(true); else LFS_EWA_EPILOGUE(false);
#undef LFS_EWA_EPILOGUE
    return check_launch("ewa_epilogue");
}

}  // namespace lfs
