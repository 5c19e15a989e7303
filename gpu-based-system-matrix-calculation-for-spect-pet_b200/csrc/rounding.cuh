// Correctly rounded float division, reciprocal and square root without range branches, for
// operands of ordinary size.  Each returns the float the IEEE operation returns (compared with
// it by tests/test_gpu_rounding.py), so code that must reproduce a float program can share a
// reciprocal between divisions and stay straight-line: the general operations each end in a
// range test and a call.
#pragma once

#include <cuda_runtime.h>

namespace sysmat {

constexpr float kMinDivisor = 1e-15f;   // div_by: smaller divisors take the IEEE division
constexpr float kMinRoot = 0x1p-100f;   // sqrt_mid: the least argument

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

// a b + c d, a b - c d and x^2 + y^2 + z^2 with the fused product written out: which product of a
// sum of two the compiler fuses depends on the code around it, so two kernels that inline the same
// function can differ in the last bit.
__device__ __forceinline__ float sum2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float diff2(float a, float b, float c, float d) { return __fmaf_rn(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ double sum2(double a, double b, double c, double d) { return __fma_rn(a, b, __dmul_rn(c, d)); }
__device__ __forceinline__ double diff2(double a, double b, double c, double d) { return __fma_rn(a, b, -__dmul_rn(c, d)); }
__device__ __forceinline__ float norm3(float x, float y, float z) { return __fmaf_rn(z, z, sum2(x, x, y, y)); }
__device__ __forceinline__ double norm3(double x, double y, double z) { return __fma_rn(z, z, sum2(x, x, y, y)); }

// Reciprocal and square root in double within about an ulp, from a float seed (relative error
// 2^-22) by Newton's method: two steps square the error twice.  For arguments whose float value is
// normal; no range branch.
__device__ __forceinline__ double rcp64(double b)
{
    double y = (double)rcp_approx((float)b);
    y = fma(y, fma(-b, y, 1.0), y);
    return fma(y, fma(-b, y, 1.0), y);
}

__device__ __forceinline__ double sqrt64(double x)
{
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)x));
    const double y = (double)f;
    const double g = x * y, h = 0.5 * y;                  // sqrt(x), 1 / (2 sqrt(x)): coupled step
    const double r = fma(-g, h, 0.5);
    const double g1 = fma(g, r, g), h1 = fma(h, r, h);
    return fma(fma(-g1, g1, x), h1, g1);
}

}  // namespace sysmat
