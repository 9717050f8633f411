// rm_approx.cuh - the blend's elementary operations that are not the language's
// own, each with the range it is used over.  tests/test_gpu_approx.py holds
// them to these bounds.
#pragma once

namespace rm {

// exp(x) = 2^(x log2 e) for x <= 0, by the approximate base-2 exponential
// (relative error at most 2^-22, results below 2^-126 are 0: PTX ISA,
// ex2.approx.ftz.f32).  The rounded exponent adds |x| 2^-23 at most.
__device__ __forceinline__ float exp_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.44269504f));
    return y;
}

// 1 / x for |x| from 1e-10 (the least |dot(n, d)| of a plane that counts) to
// 2^126, by the approximate reciprocal (relative error at most 2^-23: PTX ISA,
// rcp.approx.ftz.f32).
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// x / 3, correctly rounded for every x >= 0: the quotient by the rounded
// reciprocal, corrected once by its exact remainder (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM Journal of
// Research and Development 34(1), 1990).
__device__ __forceinline__ float third(float x) {
    const float r3 = 1.0f / 3.0f;
    const float q = x * r3;
    const float y = fmaf(fmaf(-3.0f, q, x), r3, q);
    return x <= 3.402823466e38f ? y : x;  // infinite: no remainder
}

}  // namespace rm
