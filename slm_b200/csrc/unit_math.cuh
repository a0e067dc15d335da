// unit_math.cuh -- correctly rounded square roots, reciprocals and quotients of
// vector lengths from one reciprocal square root estimate, without a test or a
// branch (the callers' guards keep the operands in range).
//
// The method is P. Markstein's ("Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990): an estimate
// is corrected by a residual that one fused operation forms exactly.  With y
// the correctly rounded reciprocal of b, q = RN(x y) and e = b q - x,
// RN(q - e y) is the correctly rounded quotient x / b.  Where y is not quite
// the rounded reciprocal, the proof still holds with
//   d (b + 2^-23) < 2^-23  and  d <= 2^-25 b (1 + 2^-18),   d = |y b - 1|,
// b scaled into [1, 2) (the first keeps the correction on the right side of a
// midpoint, the second the first quotient next to it), provided that the
// residual is exact: x is zero or at least 2^-103, the quotient normal.
// slm_selftest_unit checks both for every float a length can come from.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace slm {

constexpr uint32_t ROOT_MIN_BITS = 0x0d800000u, ROOT_MAX_BITS = 0x7f7fffffu;  // 2^-100 .. the largest float

__device__ __forceinline__ float rsqrt_estimate(float s) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    return y;
}

// y / 2 by its exponent: the float units are the busier ones
__device__ __forceinline__ float half_of(float y) { return __uint_as_float(__float_as_uint(y) - 0x800000u); }

// IEEE square root of s, given its reciprocal root's estimate y0
__device__ __forceinline__ float root_from(float s, float y0) {
    const float g = __fmul_rn(s, y0);
    return __fmaf_rn(__fmaf_rn(-g, g, s), half_of(y0), g);
}

// The reciprocal of len, given an estimate of it that comes from the square of
// len, or of a float next to it.  The bias of 2^-44 (a 2^-21 part of an ulp)
// decides the one tie that Newton's step rounds down, len = (2 - 2^-23) 2^k.
__device__ __forceinline__ float reciprocal_from(float len, float y0) {
    const float e = __fadd_rn(__fmaf_rn(-len, y0, 1.0f), 0x1p-44f);
    return __fmaf_rn(e, y0, y0);
}

// x / len with y its reciprocal; keeps a zero's sign
__device__ __forceinline__ float quotient_from(float x, float len, float y) {
    const float q = __fmul_rn(x, y);
    return __fmaf_rn(-__fmaf_rn(len, q, -x), y, q);
}

}  // namespace slm
