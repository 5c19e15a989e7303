// Correctly rounded float division, reciprocal and square root without range branches, for
// operands of ordinary size.  Each returns the float the IEEE operation returns (compared with
// it by tests/test_gpu_rounding.py), so code that must reproduce a float program can share a
// reciprocal between divisions and stay straight-line: the general operations each end in a
// range test and a call.
#pragma once

#include <cuda_runtime.h>

namespace sysmat {

constexpr float kMinDivisor = 1e-15f;   // div_by: smaller divisors take the IEEE division

// Correctly rounded a / b, given y = RN(1 / b): two residual corrections of a y.  The first
// makes the quotient faithful, and by Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990) the
// second, from a faithful quotient and a correctly rounded reciprocal, rounds correctly.  For
// finite a and normal b and y whose residuals do not underflow.
__device__ __forceinline__ float div_by(float a, float b, float y)
{
    float q = __fmul_rn(a, y);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// 1 / x within an ulp, for the geometric filters (their margins are far above it).
__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// RN(1 / b) for normal b with a normal reciprocal: two Newton steps (the second rounds
// correctly; checked against the IEEE operation for every mantissa), without a range branch.
__device__ __forceinline__ float rcp_rn(float b)
{
    float y = rcp_approx(b);
    y = __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
    return __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
}

__device__ __forceinline__ float div_rn(float a, float b) { return div_by(a, b, rcp_rn(b)); }

// Correctly rounded square root of x in [2^-100, 2^100]: one Newton step on x times the
// approximate reciprocal root, its residual exact (P. Markstein, "IA-64 and Elementary
// Functions", 2000, chapter 9; checked against the IEEE operation for every mantissa of two
// binades).  No range branch, unlike the general square root.
__device__ __forceinline__ float sqrt_mid(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float g = __fmul_rn(x, y);
    return __fmaf_rn(__fmaf_rn(-g, g, x), __fmul_rn(0.5f, y), g);
}

}  // namespace sysmat
