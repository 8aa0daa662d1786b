// What the blend kernels of both paths share: copies and approximations, the pixels of a thread (one, or two in the halves of a 64-bit register), and how the
// tiles are dealt to kernels with one pixel per thread and with two.
#pragma once

#include "common.cuh"

namespace lfs {

// 16-byte asynchronous copies to shared memory.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// One special-function instruction (relative error 2^-23); __fdividef spends four more on denominators above 2^126.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two pixels of one thread as one operand of the packed fp32 instructions (one issue slot for both, each half rounded like the
// scalar instruction). A factor that both pixels share costs nothing to replicate: in a loop of nothing else, four packed fmas with
// replicated factors take 5.9 issue slots and 0.62 of the time of the eight scalar fmas (10.5).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 both2(float a) { return pair2(a, a); }
__device__ __forceinline__ float2 halves2(f32x2 v) {
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
// The same names for one pixel, so that the kernels are written once. Pixels<PX>: what PX pixels of a thread are held in.
__device__ __forceinline__ float add2(float a, float b) { return a + b; }
__device__ __forceinline__ float mul2(float a, float b) { return a * b; }
__device__ __forceinline__ float fma2(float a, float b, float c) { return fmaf(a, b, c); }
template <int PX>
struct Pixels {
    using V = f32x2;
    static __device__ __forceinline__ V make(const float* a) { return pair2(a[0], a[1]); }
    static __device__ __forceinline__ V all(float a) { return both2(a); }
    static __device__ __forceinline__ void get(V v, float* a) { const float2 h = halves2(v); a[0] = h.x; a[1] = h.y; }
    static __device__ __forceinline__ float sum(V v) { const float2 h = halves2(v); return h.x + h.y; }
};
template <>
struct Pixels<1> {
    using V = float;
    static __device__ __forceinline__ V make(const float* a) { return a[0]; }
    static __device__ __forceinline__ V all(float a) { return a; }
    static __device__ __forceinline__ void get(V v, float* a) { a[0] = v; }
    static __device__ __forceinline__ float sum(V v) { return v; }
};

// Few tiles can carry a large image (a distant object, the inset of a lens), and then the walk of the longest lists is what a kernel with two pixels per thread takes.
// Lists that hold more than one in `share` of all instances are left to a launch with one pixel per thread, twice the warps, beside the other one. Forward +
// backward of 200 k and 1.5 M Gaussians in us at 1920x1080, with two pixels everywhere and now: seen on some 64 tiles 318 + 322 and 142 + 218, 1014 + 970 and 752 + 688,
// on 30 tiles 752 + 700 and 412 + 341, 3239 + 3056 and 1469 + 989; EWA, 30 tiles 705 + 725 and 458 + 437, 2896 + 3598 and 1817 + 1850. Where no list is that
// long the second launch costs 1 to 2 us. On an image of few tiles lists of several times the mean are common, and the launch with two pixels has the cheaper
// sums: there a list counts from one in half an SM on (EWA backward of 1.2 M on 858 tiles, 299 us: 333 with one in 107).
struct Outsized { int share, slots; };   // slots: tiles that may have an outsized list, from the start of the launch order
inline Outsized outsized_lists(const int32_t* tile_order, int n_tiles) {
    // without an order (operators) the second launch would have to look at every tile: 10 us beside 350, 1.0 M on 5,922 tiles 14 beside 445 and 17 beside 895
    if (!tile_order) return Outsized{};
    const int share = n_tiles >= 16 * num_sms() ? 3 * num_sms() : num_sms() / 2;
    // fewer than `share` lists are outsized, and at most a quarter as many others come before the last of them, since the order tells lengths apart by quarters
    // of a power of two
    const int slots = share + share / 4 + 1;
    return Outsized{share, n_tiles < slots ? n_tiles : slots};
}
__device__ __forceinline__ bool is_outsized(int32_t n, int32_t n_isects, const Outsized& o) { return (int64_t)n * o.share > n_isects; }
// First thing in both kernels of such a pair; either also runs alone, with share = 0.
template <int PX>
__device__ __forceinline__ void side_by_side(const Outsized& o) {
    if (PX == 1) { if (o.share) let_next_start(); }
    else if (blockIdx.x == gridDim.x - 1) wait_for_previous();
}

}  // namespace lfs
