// sf_divide.cuh -- the update's division by 6 (pressure) or 1 + 6 alpha
// (diffusion) in FP32, for kernels whose instruction count matters.
//
// tb::divide (sf_stencil_tb.cuh) forms the quotient in FP64, whatever the
// numerator. Away from the ends of the FP32 range the same correction works in
// FP32: q = RN(n y) with y = RN(1 / d), r = n - q d (exact with an FMA),
// q' = RN(q + r y). Markstein's theorem (IBM J. Res. Dev. 34(1), 1990) makes
// q' the correctly rounded quotient when q is faithful; one correction makes q
// faithful for any d, a second one rounds it. For d = 6 the first correction
// alone is right for all 2^23 significands (checked exhaustively by
// tests/test_resident.py). The remainders are exact while no bit of q d falls
// below 2^-149 and nothing overflows, which easy() ensures:
// 2^-98 <= |n| <= 2^126 with 1 <= d <= 2^20. Zeros give zeros. Everything else
// (tiny numerators in the far field of a plume, infinities, NaN, other d)
// takes tb::divide.
#pragma once

#include "sf_f32x2.cuh"
#include "sf_stencil_tb.cuh"

namespace sfb::divide {

struct Divisor {
    float d, y;   // the divisor and RN32(1 / d)
    float lo;     // smallest |n| of the FP32 form
    double y64;   // RN64(1 / d), for tb::divide
};

__device__ __forceinline__ Divisor make_divisor(float d) {
    Divisor v;
    v.d = d;
    v.y = __frcp_rn(d);
    v.lo = d >= 1.0f && d <= 0x1p20f ? 0x1p-98f : __int_as_float(0x7f800000);
    v.y64 = tb::recip64(d);
    return v;
}

// All four numerators suit the FP32 form. A NaN among them passes (fmaxf and
// fminf drop it), which gives a NaN either way; zeros do not pass.
__device__ __forceinline__ bool easy(float4 n, const Divisor& v) {
    const float big = fmaxf(fmaxf(fabsf(n.x), fabsf(n.y)), fmaxf(fabsf(n.z), fabsf(n.w)));
    const float small = fminf(fminf(fabsf(n.x), fabsf(n.y)), fminf(fabsf(n.z), fabsf(n.w)));
    return small >= v.lo && big <= 0x1p126f;
}

// RN(n / d) for an n, or a pair, that easy() allows.
template <bool SIX>
__device__ __forceinline__ float quotient(float n, const Divisor& v) {
    const float q0 = __fmul_rn(n, v.y);
    const float q1 = __fmaf_rn(__fmaf_rn(-q0, v.d, n), v.y, q0);
    if constexpr (SIX) return q1;
    return __fmaf_rn(__fmaf_rn(-q1, v.d, n), v.y, q1);
}
template <bool SIX>
__device__ __forceinline__ F2 quotient(F2 n, const Divisor& v) {
    const F2 y = f2(v.y, v.y), d = f2(-v.d, -v.d);
    const F2 q0 = n * y;
    const F2 q1 = fma2(fma2(q0, d, n), y, q0);
    if constexpr (SIX) return q1;
    return fma2(fma2(q1, d, n), y, q1);
}

// RN(n / d) for four numerators, any of them.
__device__ __forceinline__ float4 hard(float4 n, const Divisor& v) {
    if (n.x == 0.0f && n.y == 0.0f && n.z == 0.0f && n.w == 0.0f) return n;  // the far field
    return make_float4(tb::divide(n.x, v.d, v.y64), tb::divide(n.y, v.d, v.y64), tb::divide(n.z, v.d, v.y64), tb::divide(n.w, v.d, v.y64));
}

// The same, the FP32 form where it serves; SIX: d is 6.
template <bool SIX>
__device__ __forceinline__ float4 four(float4 n, const Divisor& v) {
    if (easy(n, v)) [[likely]] {
        const F4 p = f4(n);
        return unpack(F4{quotient<SIX>(p.lo, v), quotient<SIX>(p.hi, v)});
    }
    return hard(n, v);
}

}  // namespace sfb::divide
