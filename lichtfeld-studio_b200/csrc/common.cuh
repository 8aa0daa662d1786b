// Shared declarations of the lfs_b200 CUDA library (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lfs_b200.h"

namespace lfs {

// ---------------------------------------------------------------------------------------------
// Error reporting: every entry point returns a status and leaves a message for lfs_last_error().
// ---------------------------------------------------------------------------------------------
void set_error(const char* fmt, ...);
int check_launch(const char* what);

// Opt-in per-kernel timing (lfs_profile_enable): when on, a KernelTimer brackets a launch with two
// CUDA events on the launching stream; lfs_profile_collect returns the elapsed times. With the NVTX bit it opens an
// NVTX range of the same name around the launch for timeline tools. Off by default and free when off.
struct KernelTimer {
    KernelTimer(const char* name, cudaStream_t st);
    ~KernelTimer();
    const char* name_;
    cudaStream_t st_;
    void* a_;
    void* b_;
    bool nvtx_;
};
#define LFS_TIMED(name, st) ::lfs::KernelTimer lfs_kernel_timer_(name, st)

#define LFS_REQUIRE(cond, msg)                         \
    do {                                               \
        if (!(cond)) {                                 \
            ::lfs::set_error("%s: %s", __func__, msg); \
            return LFS_EINVAL;                         \
        }                                              \
    } while (0)

// Persistent / grid-stride kernels are sized in multiples of the SM count of the current device (148 on a B200),
// read once per device from cudaDevAttrMultiProcessorCount.
int num_sms();

inline int grid_for(int64_t n, int block, int max_blocks_per_sm = 8) {
    int64_t g = (n + block - 1) / block;
    const int64_t cap = (int64_t)num_sms() * max_blocks_per_sm;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

template <class... P, class... A>
void launch(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) { kernel<<<grid, block, smem, st>>>(args...); }
// A launch that starts as soon as every CTA of the launch before it has called let_next_start() or has ended. That launch has to have started behind everything
// the new one reads, and one thread of the new one calls wait_for_previous(), so that what comes after it comes after both.
template <class... P, class... A>
void launch_beside(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute beside;
    beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    beside.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = &beside; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// Per-camera constants derived once per call by camera_setup_kernel from the row-major
// world-to-camera matrix and the intrinsics (global shutter).
// ---------------------------------------------------------------------------------------------
struct CamDev {
    float qw, qx, qy, qz;  // quat_cast of the rotation block
    float tx, ty, tz;      // translation column
    float Rinv[9];         // mat3_cast(inverse(q)), row-major
    float ro[3];           // world ray origin = -Rinv * t
    float campos[3];       // -R^T t (what inverse(viewmat)[:3,3] gives), used for SH directions
    float fx, fy, cx, cy;
    float k[4];            // fisheye radial coefficients
    float dist[12];        // OpenCV pinhole distortion: k1..k6, p1, p2, s1..s4 (model == LFS_PINHOLE_OPENCV)
    float max_angle;       // fisheye
    float approx_b1;       // fisheye: linear term of the crude backward polynomial
    int W, H, model;
    int rs_type;           // ShutterType of the reference: 0..3 rolling (top-to-bottom, left-to-right, bottom-to-top,
                           // right-to-left), 4 global
    // rolling shutter: end-of-frame pose (equal to the start pose without one) and the centre-of-frame pose that
    // gives the depth of a Gaussian (gsplat/ProjectionUT3DGSFused.cu:73-77)
    int has_end;
    float q1w, q1x, q1y, q1z, t1x, t1y, t1z;
    float qcw, qcx, qcy, qcz, tcx, tcy, tcz;
};
constexpr int LFS_SHUTTER_GLOBAL = 4;

// Internal model id: LFS_PINHOLE with any of the three distortion tensors present selects the OpenCV pinhole
// model (gsplat/ProjectionUT3DGSFused.cu:91-113); it never crosses the C ABI.
constexpr int LFS_PINHOLE_OPENCV = 4;
inline int effective_model(int model, const float* radial, const float* tangential, const float* thin_prism) {
    return (model == LFS_PINHOLE && (radial || tangential || thin_prism)) ? LFS_PINHOLE_OPENCV : model;
}

// One packed 64-byte record per Gaussian for the rasterizer. Cameras with one ray origin (global shutter), d = the pixel's
// camera-space direction, (e1, e2, w) = (p1, p2, p3) . d, phi = (e1^2 + e2^2) / (e1^2 + e2^2 + w^2) (RayFrame in gsmath.cuh):
//   r0 = (p1, c)              c = -|g|^2 log2(e) / 2: the response is exp2(c phi)
//   r1 = (p2, phi_cut)        p2.x = 0 for the planar models (pinhole, OpenCV); alpha < 1/255 for certain when phi > phi_cut
//   r2 = (p3, alpha_cut)      alpha >= 1/255 for certain when it is not below alpha_cut
//   r3 = (red, green, blue, opacity)
// Between the two cuts the pair is decided by the product form |u x g|^2 / |u|^2, u = M d, from the cut record
//   c0 .. c2 = rows of M = diag(1/scale) R^T, each followed by its element of g = M (ray origin - mean)
// Rolling shutter, where the ray origin differs from pixel to pixel:
//   r0 .. r2 = rows of M = diag(1/scale) R^T, each followed by its element of gro = M (start-pose origin - mean); r3 as above
constexpr int kRecordFloats = 16;

// Host-side launchers shared between translation units (all asynchronous on `st`).
// radial: [C,4] for LFS_FISHEYE, [C,6] for LFS_PINHOLE; tangential [C,2] and thin_prism [C,4] only for LFS_PINHOLE.
// viewmats1 [C,4,4] or null (no end pose), rs_type = ShutterType (4 = global)
int launch_camera_setup(int C, const float* viewmats, const float* viewmats1, int rs_type, const float* Ks, const float* radial,
                        const float* tangential, const float* thin_prism, int W, int H, int model, CamDev* cams,
                        cudaStream_t st);

// Instances per tile, and where the next one goes. The counters exist `replicas` times (a power of two), `stride` apart; the Gaussians
// g .. g + 31, g a multiple of 32, use the same ones when they are counted and when they are written.
struct TileCounters {
    int32_t *counts, *cursors;
    int32_t replicas, stride;
    __device__ __forceinline__ size_t replica(int64_t g) const { return (size_t)((g >> 5) & (replicas - 1)) * stride; }
};

// ---- sort.cu -------------------------------------------------------------------------------
struct SortScratch {
    uint32_t* block_sums; // [kScanBlocks + 1]
};
// Capacity of the scratch array; the launches use min(4 x SM count, capacity) blocks.
constexpr int kScanBlocks = 1024;

// out[i] = exclusive prefix sum of src; total written to *total_dev.
int exclusive_scan(const int32_t* src, int64_t n, int32_t* out, int32_t* total_dev, const SortScratch& scratch, cudaStream_t st);

// One 16-byte store to an NVSwitch multicast address: the switch writes it into the same offset of every GPU bound to the
// multicast object (this GPU included), so a broadcast leaves this GPU's NVLink ports once instead of once per peer.
__device__ __forceinline__ void multimem_st4(float* mc, const float4 v) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
__device__ __forceinline__ void multimem_st1(float* mc, const float v) {
    asm volatile("multimem.st.relaxed.sys.global.f32 [%0], %1;" ::"l"(mc), "f"(v) : "memory");
}

}  // namespace lfs
