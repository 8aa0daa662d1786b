// Separable 11x11 Gaussian-window SSIM (forward with derivative maps, backward) and the fused
// photometric loss 0.8 L1 + 0.2 (1 - SSIM_valid) with its gradient w.r.t. the unclamped HWC render.
//
// Replaces src/training/kernels/ssim.cu:64 (K9) and :284 (K10), the crop / pad / mean glue of
// include/kernels/fused_ssim.cuh:59-67, :85-96, :117-122, torch::l1_loss of
// src/training/trainer.cpp:126 and the clamp + permute of src/training/rasterization/rasterizer.cpp:205.
// Stencil work, bound by instruction issue and shared-memory accesses: each CTA stages the 42x42 halo tile of a 32x32 output
// tile of one channel in shared memory and runs the 11-tap horizontal and vertical passes from register windows. The planes
// that are filtered alike are kept as pairs (x, y), (x^2, y^2) and filtered two at a time with the packed fp32 instructions
// (one issue slot and one 8-byte shared load for both, each element rounded as by the scalar instruction). 352 threads: the
// 42 rows x 8 column groups of the horizontal pass and the 32 columns x 11 strips of the vertical pass each fill them once.
#include "common.cuh"
#include "loss.cuh"

namespace lfs {

namespace {

constexpr int kT = 32;             // output tile edge
constexpr int kHalo = 5;
constexpr int kS = kT + 2 * kHalo;   // 42: halo tile edge
constexpr int kSX = kS + 1;          // 43: row stride of the staged images (conflict-free for lanes that walk rows)
constexpr int kSH = kT + 1;          // 33: row stride of the horizontally filtered planes
constexpr int kThreadsLoss = 352;
constexpr int kColGroups = kT / 4;   // a horizontal work item filters 4 adjacent columns of one row
constexpr int kStrip = 3;            // a vertical work item filters 3 stacked rows of one column
static_assert(kS * kColGroups <= kThreadsLoss && kThreadsLoss / 32 * kStrip >= kT, "one round per pass");

__constant__ float cTaps[11] = {
    0.001028380123898387f, 0.0075987582094967365f, 0.036000773310661316f, 0.10936068743467331f,
    0.21300552785396576f,  0.26601171493530273f,   0.21300552785396576f,  0.10936068743467331f,
    0.036000773310661316f, 0.0075987582094967365f, 0.001028380123898387f};

// FUSED: img1 is the unclamped HWC render (clamped to [0,1] on load); otherwise plain CHW.
template <bool FUSED>
__device__ __forceinline__ float load_img1(const float* img1, int c, int y, int x, int H, int W) {
    if (x < 0 || x >= W || y < 0 || y >= H) return 0.f;
    if (FUSED) return fminf(1.f, fmaxf(0.f, img1[((size_t)y * W + x) * 3 + c]));
    return img1[(size_t)c * H * W + (size_t)y * W + x];
}
__device__ __forceinline__ float load_chw(const float* img, int c, int y, int x, int H, int W) {
    if (x < 0 || x >= W || y < 0 || y >= H) return 0.f;
    return img[(size_t)c * H * W + (size_t)y * W + x];
}

// 11-tap filter at centre index ci of a register window, symmetric pairs first (the reference's order of additions)
__device__ __forceinline__ float tap11(const float* v, int ci) {
    float a = 0.f;
#pragma unroll
    for (int d = 1; d <= kHalo; ++d) a += (v[ci - d] + v[ci + d]) * cTaps[kHalo - d];
    return a + v[ci] * cTaps[kHalo];
}

// Two fp32 values in one register pair.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// tap11 on pairs, the same operations on both elements; taps = the six distinct weights, each in both halves
__device__ __forceinline__ f32x2 tap11x2(const f32x2* v, int ci, const f32x2* taps) {
    f32x2 a = mul2(add2(v[ci - 1], v[ci + 1]), taps[kHalo - 1]);
#pragma unroll
    for (int d = 2; d <= kHalo; ++d) a = fma2(add2(v[ci - d], v[ci + d]), taps[kHalo - d], a);
    return fma2(v[ci], taps[kHalo], a);
}

// One CTA filters a 32x32 output tile of one channel (blockIdx.z). The 42x42 halo tile is staged in shared memory;
// the horizontal pass gives every thread 4 adjacent outputs of one row from a 14-value register window, the vertical pass 3
// stacked outputs of one column from 13-value windows of the filtered planes.
//
// Forward. Plain mode writes ssim_map and the three derivative maps. Fused mode writes the derivative maps already
// multiplied by dL/dmap (map_grad inside the valid crop, 0 outside) and accumulates sum(ssim over the crop) and
// sum(|img1 - img2|) into sums[0], sums[1].
template <bool FUSED>
__global__ void __launch_bounds__(kThreadsLoss, 3) ssim_fwd_kernel(int CH, int H, int W, float C1, float C2,
                                                                  const float* __restrict__ img1, const float* __restrict__ img2,
                                                                  float* __restrict__ ssim_map, float* __restrict__ dm_dmu1,
                                                                  float* __restrict__ dm_dsigma1_sq, float* __restrict__ dm_dsigma12,
                                                                  float map_grad, int crop, double* __restrict__ sums) {
    __shared__ f32x2 sXY[kS][kSX];            // (img1, img2)
    __shared__ f32x2 sM[kS][kSH], sQ[kS][kSH];  // filtered (x, y) and (x^2, y^2)
    __shared__ float sP[kS][kSH];               // filtered x y
    __shared__ float red[2][kThreadsLoss / 32];
    const int tid = threadIdx.x, c = blockIdx.z;
    const int bx0 = blockIdx.x * kT, by0 = blockIdx.y * kT;
    f32x2 taps[kHalo + 1];
#pragma unroll
    for (int d = 0; d <= kHalo; ++d) taps[d] = pack2(cTaps[d], cTaps[d]);
    for (int q = tid; q < kS * kS; q += kThreadsLoss) {
        const int ly = q / kS, lx = q - ly * kS;
        sXY[ly][lx] = pack2(load_img1<FUSED>(img1, c, by0 + ly - kHalo, bx0 + lx - kHalo, H, W),
                            load_chw(img2, c, by0 + ly - kHalo, bx0 + lx - kHalo, H, W));
    }
    __syncthreads();
    if (tid < kS * kColGroups) {
        const int cg = tid / kS, row = tid - cg * kS;
        f32x2 w[14];
        float xy[14];
#pragma unroll
        for (int j = 0; j < 14; ++j) {
            w[j] = sXY[row][cg * 4 + j];
            const float2 v = unpack2(w[j]);
            xy[j] = v.x * v.y;
        }
#pragma unroll
        for (int o = 0; o < 4; ++o) sP[row][cg * 4 + o] = tap11(xy, o + kHalo);
#pragma unroll
        for (int o = 0; o < 4; ++o) sM[row][cg * 4 + o] = tap11x2(w, o + kHalo, taps);
#pragma unroll
        for (int j = 0; j < 14; ++j) w[j] = mul2(w[j], w[j]);
#pragma unroll
        for (int o = 0; o < 4; ++o) sQ[row][cg * 4 + o] = tap11x2(w, o + kHalo, taps);
    }
    __syncthreads();
    const int col = tid & 31, strip = (tid >> 5) * kStrip;
    float2 mu[kStrip], sq[kStrip];
    float sxy[kStrip];
    constexpr int kWin = kStrip + 2 * kHalo;
    {
        // windows past the last strip read the last row again; those outputs lie outside the tile
        f32x2 h[kWin];
#pragma unroll
        for (int j = 0; j < kWin; ++j) h[j] = sM[min(strip + j, kS - 1)][col];
#pragma unroll
        for (int o = 0; o < kStrip; ++o) mu[o] = unpack2(tap11x2(h, o + kHalo, taps));
#pragma unroll
        for (int j = 0; j < kWin; ++j) h[j] = sQ[min(strip + j, kS - 1)][col];
#pragma unroll
        for (int o = 0; o < kStrip; ++o) sq[o] = unpack2(tap11x2(h, o + kHalo, taps));
        float g[kWin];
#pragma unroll
        for (int j = 0; j < kWin; ++j) g[j] = sP[min(strip + j, kS - 1)][col];
#pragma unroll
        for (int o = 0; o < kStrip; ++o) sxy[o] = tap11(g, o + kHalo);
    }
    float ssim_acc = 0.f, l1_acc = 0.f;
    const int x = bx0 + col;
#pragma unroll
    for (int o = 0; o < kStrip; ++o) {
        const int y = by0 + strip + o;
        if (strip + o < kT && x < W && y < H) {
            const float mu1 = mu[o].x, mu2 = mu[o].y;
            const float mu1_sq = mu1 * mu1, mu2_sq = mu2 * mu2;
            const float sigma1_sq = sq[o].x - mu1_sq, sigma2_sq = sq[o].y - mu2_sq, sigma12 = sxy[o] - mu1 * mu2;
            const float A = mu1_sq + mu2_sq + C1, B = sigma1_sq + sigma2_sq + C2;
            const float C_ = 2.f * mu1 * mu2 + C1, D_ = 2.f * sigma12 + C2;
            // two divisions serve the map and its derivatives
            const float rA = 1.0f / A, rB = 1.0f / B;
            const float cA = C_ * rA, dB = D_ * rB;
            const float val = cA * dB;
            const float g_mu1 = 2.f * (mu2 * rA * dB - mu2 * rB * cA - mu1 * rA * val + mu1 * rB * val);
            const float g_s1 = -val * rB;
            const float g_s12 = 2.f * cA * rB;
            const size_t gi = (size_t)c * H * W + (size_t)y * W + x;
            if (FUSED) {
                const bool in_crop = !crop || (x >= kHalo && x < W - kHalo && y >= kHalo && y < H - kHalo);
                const float chain = in_crop ? map_grad : 0.f;
                dm_dmu1[gi] = g_mu1 * chain;
                dm_dsigma1_sq[gi] = g_s1 * chain;
                dm_dsigma12[gi] = g_s12 * chain;
                if (in_crop) ssim_acc += val;
                const float2 v = unpack2(sXY[strip + o + kHalo][col + kHalo]);
                l1_acc += fabsf(v.x - v.y);
            } else {
                ssim_map[gi] = val;
                if (dm_dmu1) { dm_dmu1[gi] = g_mu1; dm_dsigma1_sq[gi] = g_s1; dm_dsigma12[gi] = g_s12; }
            }
        }
    }
    if (FUSED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ssim_acc += __shfl_xor_sync(0xffffffffu, ssim_acc, o);
            l1_acc += __shfl_xor_sync(0xffffffffu, l1_acc, o);
        }
        if ((tid & 31) == 0) { red[0][tid >> 5] = ssim_acc; red[1][tid >> 5] = l1_acc; }
        __syncthreads();
        if (tid == 0) {
            double s_ = 0.0, l_ = 0.0;
            for (int k = 0; k < kThreadsLoss / 32; ++k) { s_ += red[0][k]; l_ += red[1][k]; }
            atomicAdd(&sums[0], s_);
            atomicAdd(&sums[1], l_);
        }
    }
}

// Backward, same tiling. Plain mode: maps are multiplied by dL_dmap on load and dL_dimg1 is CHW. Fused mode: the maps
// are pre-multiplied, the L1 sign term and the clamp mask are applied and the output is the HWC gradient of the
// unclamped render, scaled by grad_scale.
template <bool FUSED>
__global__ void __launch_bounds__(kThreadsLoss, 4) ssim_bwd_kernel(int CH, int H, int W, const float* __restrict__ img1,
                                                                  const float* __restrict__ img2, const float* __restrict__ dL_dmap,
                                                                  const float* __restrict__ dm_dmu1, const float* __restrict__ dm_dsigma1_sq,
                                                                  const float* __restrict__ dm_dsigma12, float* __restrict__ dL_dimg1,
                                                                  float l1_grad, float grad_scale) {
    __shared__ f32x2 sD[kS][kSX];    // (d mu1, d sigma1^2)
    __shared__ float sE[kS][kSX];    // d sigma12
    __shared__ f32x2 sHD[kS][kSH];
    __shared__ float sHE[kS][kSH];
    const int tid = threadIdx.x, c = blockIdx.z;
    const int bx0 = blockIdx.x * kT, by0 = blockIdx.y * kT;
    f32x2 taps[kHalo + 1];
#pragma unroll
    for (int d = 0; d <= kHalo; ++d) taps[d] = pack2(cTaps[d], cTaps[d]);
    for (int q = tid; q < kS * kS; q += kThreadsLoss) {
        const int ly = q / kS, lx = q - ly * kS;
        const int gy = by0 + ly - kHalo, gx = bx0 + lx - kHalo;
        const float chain = FUSED ? 1.f : load_chw(dL_dmap, c, gy, gx, H, W);
        sD[ly][lx] = pack2(load_chw(dm_dmu1, c, gy, gx, H, W) * chain, load_chw(dm_dsigma1_sq, c, gy, gx, H, W) * chain);
        sE[ly][lx] = load_chw(dm_dsigma12, c, gy, gx, H, W) * chain;
    }
    __syncthreads();
    if (tid < kS * kColGroups) {
        const int cg = tid / kS, row = tid - cg * kS;
        f32x2 w[14];
#pragma unroll
        for (int j = 0; j < 14; ++j) w[j] = sD[row][cg * 4 + j];
#pragma unroll
        for (int o = 0; o < 4; ++o) sHD[row][cg * 4 + o] = tap11x2(w, o + kHalo, taps);
        float v[14];
#pragma unroll
        for (int j = 0; j < 14; ++j) v[j] = sE[row][cg * 4 + j];
#pragma unroll
        for (int o = 0; o < 4; ++o) sHE[row][cg * 4 + o] = tap11(v, o + kHalo);
    }
    __syncthreads();
    const int col = tid & 31, strip = (tid >> 5) * kStrip;
    constexpr int kWin = kStrip + 2 * kHalo;
    float2 s01[kStrip];
    float s2[kStrip];
    {
        f32x2 h[kWin];
#pragma unroll
        for (int j = 0; j < kWin; ++j) h[j] = sHD[min(strip + j, kS - 1)][col];
#pragma unroll
        for (int o = 0; o < kStrip; ++o) s01[o] = unpack2(tap11x2(h, o + kHalo, taps));
        float g[kWin];
#pragma unroll
        for (int j = 0; j < kWin; ++j) g[j] = sHE[min(strip + j, kS - 1)][col];
#pragma unroll
        for (int o = 0; o < kStrip; ++o) s2[o] = tap11(g, o + kHalo);
    }
    const int x = bx0 + col;
#pragma unroll
    for (int o = 0; o < kStrip; ++o) {
        const int y = by0 + strip + o;
        if (strip + o < kT && x < W && y < H) {
            if (FUSED) {
                const float raw = img1[((size_t)y * W + x) * 3 + c];
                const float p1 = fminf(1.f, fmaxf(0.f, raw));
                const float p2 = img2[(size_t)c * H * W + (size_t)y * W + x];
                float g = s01[o].x + (2.f * p1) * s01[o].y + (p2)*s2[o];
                const float diff = p1 - p2;
                g += l1_grad * (diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f));
                if (!(raw >= 0.f && raw <= 1.f)) g = 0.f;
                dL_dimg1[((size_t)y * W + x) * 3 + c] = g * grad_scale;
            } else {
                const size_t gi = (size_t)c * H * W + (size_t)y * W + x;
                const float p1 = img1[gi], p2 = img2[gi];
                dL_dimg1[gi] = s01[o].x + (2.f * p1) * s01[o].y + (p2)*s2[o];
            }
        }
    }
}

__global__ void loss_finalize_kernel(const double* sums, double n_all, double n_valid, float lambda, float* loss) {
    const float l1 = (float)(sums[1] / n_all);
    const float ssim = (float)(sums[0] / n_valid);
    loss[0] = (1.f - lambda) * l1 + lambda * (1.f - ssim);
    loss[1] = l1;
    loss[2] = ssim;
}

}  // namespace

int launch_fusedssim(int CH, int H, int W, float C1, float C2, const float* img1, const float* img2, float* ssim_map,
                     float* dm1, float* ds1, float* ds12, cudaStream_t st) {
    if (CH * H * W == 0) return LFS_OK;
    dim3 grid((W + kT - 1) / kT, (H + kT - 1) / kT, CH), block(kThreadsLoss);
    ssim_fwd_kernel<false><<<grid, block, 0, st>>>(CH, H, W, C1, C2, img1, img2, ssim_map, dm1, ds1, ds12, 0.f, 0, nullptr);
    return check_launch("fusedssim");
}

int launch_fusedssim_backward(int CH, int H, int W, const float* img1, const float* img2, const float* dL_dmap,
                              const float* dm1, const float* ds1, const float* ds12, float* dL_dimg1, cudaStream_t st) {
    if (CH * H * W == 0) return LFS_OK;
    dim3 grid((W + kT - 1) / kT, (H + kT - 1) / kT, CH), block(kThreadsLoss);
    ssim_bwd_kernel<false><<<grid, block, 0, st>>>(CH, H, W, img1, img2, dL_dmap, dm1, ds1, ds12, dL_dimg1, 0.f, 1.f);
    return check_launch("fusedssim_backward");
}

namespace {
// out[c] += sum over pixels of v_render[p, c] * (1 - alpha[p]); one double atomic per CTA and channel.
__global__ void __launch_bounds__(256) background_gradient_kernel(int64_t P, int CH, const float* __restrict__ v_render,
                                                                  const float* __restrict__ alpha, double* __restrict__ acc) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < P; p += (int64_t)gridDim.x * blockDim.x) {
        const float w = 1.0f - alpha[p];
        for (int c = 0; c < CH; ++c) s[c] += (double)(v_render[p * CH + c] * w);
    }
    __shared__ double red[8][4];
    for (int c = 0; c < CH; ++c) {
        double v = s[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = v;
    }
    __syncthreads();
    if (threadIdx.x < CH) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
        atomicAdd(acc + threadIdx.x, v);
    }
}
__global__ void background_gradient_finalize_kernel(int CH, const double* __restrict__ acc, float* __restrict__ out) {
    if (threadIdx.x < CH) out[threadIdx.x] = (float)acc[threadIdx.x];
}
}  // namespace

int launch_background_gradient(int H, int W, int CH, const float* v_render, const float* alpha, float* v_background,
                               void* workspace, cudaStream_t st) {
    double* acc = reinterpret_cast<double*>(workspace);
    cudaMemsetAsync(acc, 0, 4 * sizeof(double), st);
    const int64_t P = (int64_t)H * W;
    if (P > 0) {
        LFS_TIMED("background_gradient", st);
        background_gradient_kernel<<<grid_for(P, 256, 4), 256, 0, st>>>(P, CH, v_render, alpha, acc);
    }
    background_gradient_finalize_kernel<<<1, 32, 0, st>>>(CH, acc, v_background);
    return check_launch("background_gradient");
}

size_t photometric_workspace_bytes(int H, int W) { return 256 + (size_t)3 * 3 * H * W * sizeof(float); }

int launch_photometric_loss(int H, int W, float lambda, float grad_scale, const float* render_hwc, const float* target_chw,
                            float* v_render_hwc, float* loss_dev, void* workspace, cudaStream_t st) {
    double* sums = reinterpret_cast<double*>(workspace);
    float* maps = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 256);
    const size_t plane = (size_t)3 * H * W;
    float *d1 = maps, *d2 = maps + plane, *d3 = maps + 2 * plane;
    const int crop = (H > 10 && W > 10) ? 1 : 0;
    const double n_all = 3.0 * H * W;
    const double n_valid = crop ? 3.0 * (H - 10) * (W - 10) : n_all;
    const float map_grad = (float)(-(double)lambda / n_valid);
    const float l1_grad = (float)((1.0 - (double)lambda) / n_all);
    cudaMemsetAsync(sums, 0, 2 * sizeof(double), st);
    dim3 grid((W + kT - 1) / kT, (H + kT - 1) / kT, 3), block(kThreadsLoss);
    {
    LFS_TIMED("loss_fwd", st);
    ssim_fwd_kernel<true><<<grid, block, 0, st>>>(3, H, W, (float)(0.01 * 0.01), (float)(0.03 * 0.03), render_hwc,
                                                  target_chw, nullptr, d1, d2, d3, map_grad, crop, sums);
    }
    if (v_render_hwc) {
        LFS_TIMED("loss_bwd", st);
        ssim_bwd_kernel<true><<<grid, block, 0, st>>>(3, H, W, render_hwc, target_chw, nullptr, d1, d2, d3, v_render_hwc,
                                                      l1_grad, grad_scale);
    }
    loss_finalize_kernel<<<1, 1, 0, st>>>(sums, n_all, n_valid, lambda, loss_dev);
    return check_launch("photometric_loss");
}

}  // namespace lfs
