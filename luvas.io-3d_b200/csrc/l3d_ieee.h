/*
 * Correctly rounded FP32 reciprocal and quotient for operands in a known range, on the device.
 *
 * The bit-exact kernels divide once per window sample or voxel, always by a camera depth.  The
 * general 1.0f / x has to handle subnormal, infinite and huge operands, which costs it a branch
 * that ends the straight line in which a window's samples overlap.  Here the range is the caller's
 * promise and the value is the same:
 *   reciprocal  one Newton step on the hardware approximation y (error at most one ulp):
 *               y + y (1 - x y), both operations fused.  Markstein ("Computation of elementary
 *               functions on the IBM RISC System/6000 processor", IBM J. R&D 34, 1990) shows that
 *               the step rounds correctly but for a divisor of all-ones mantissa; those come out
 *               right too: over every float of the range it equals 1.0f / x (tests/test_ieee_gpu.py).
 *   quotient    his theorem for a / b from a correctly rounded reciprocal: q = a y, then
 *               q + y (a - b q), the remainder exact.
 */
#ifndef L3D_IEEE_H
#define L3D_IEEE_H

#include <cuda_runtime.h>

/* 1.0f / x within one ulp (subnormal results are flushed). */
__device__ __forceinline__ float l3d_rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* 1.0f / x for 2^-126 <= |x| <= 2^125 (the reciprocal stays a normal number). */
__device__ __forceinline__ float l3d_rcp_normal(float x) {
    const float y = l3d_rcp_approx(x);
    return fmaf(y, fmaf(-x, y, 1.0f), y);
}

/* a / b for b as above and a zero or |a| >= 2^-100, |a / b| in [2^-100, 2^100] (no step of the
 * computation leaves the normal numbers). */
__device__ __forceinline__ float l3d_div_normal(float a, float b) {
    const float y = l3d_rcp_normal(b);
    const float q = a * y;
    return fmaf(fmaf(-b, q, a), y, q);
}

/* a / b, given y = 1.0f / b rounded, under the conditions of l3d_div_normal (a zero a excepted when its
 * sign matters: -0 / b gives +0). */
__device__ __forceinline__ float l3d_div_by(float a, float b, float y) {
    const float q = a * y;
    return fmaf(fmaf(-b, q, a), y, q);
}

/* rintf(x) as an index: for an integer n <= 2^22, the result is below n exactly when rintf(x) (ties to
 * even) lies in [0, n), and is then rintf(x).  Adding 1.5 x 2^23 leaves the rounded integer in the sum's
 * low bits; a sum outside [1.5 x 2^23, 1.5 x 2^23 + n), NaN included, has bits outside theirs. */
__device__ __forceinline__ unsigned l3d_rint_index(float x) {
    return __float_as_uint(x + 12582912.0f) - 0x4b400000u;
}

#endif
