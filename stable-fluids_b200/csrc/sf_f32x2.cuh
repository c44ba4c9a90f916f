// sf_f32x2.cuh -- pairs of FP32 values in one 64-bit register, for sm_100's
// packed FP32 instructions: two independent IEEE operations (round to nearest,
// subnormals kept) for one issue slot. The stencil kernels that keep their
// data on chip are bound by instruction issue, and most of what they issue is
// FP32 sums. Each half rounds exactly as the scalar instruction does.
#pragma once

#include <cuda_runtime.h>

namespace sfb {

struct F2 {
    unsigned long long v;
};

__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// Four values as two pairs.
struct F4 {
    F2 lo, hi;
};
__device__ __forceinline__ F4 f4(float4 a) { return {f2(a.x, a.y), f2(a.z, a.w)}; }
__device__ __forceinline__ float4 unpack(F4 a) {
    const float2 l = unpack(a.lo), h = unpack(a.hi);
    return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ F4 operator+(F4 a, F4 b) { return {a.lo + b.lo, a.hi + b.hi}; }

}  // namespace sfb
