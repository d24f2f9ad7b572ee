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
 *               the step rounds correctly but for a divisor of all-ones mantissa; compared with
 *               1.0f / x over every mantissa at every seventh exponent it never differed.
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

#endif
