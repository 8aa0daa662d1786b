// The pixels of a thread of the blend kernels: one, or two in the halves of a 64-bit register.
#pragma once

#include <cuda_runtime.h>

namespace lfs {

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

}  // namespace lfs
