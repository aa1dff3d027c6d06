// Correctly rounded float division by a divisor whose reciprocal is known, for host and device.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define PB_DIVIDE_FN __host__ __device__ __forceinline__
#else
#define PB_DIVIDE_FN inline
#endif

namespace pb {

// a / d, correctly rounded, from d and y = 1 / d correctly rounded.  Markstein (Computation of
// elementary functions on the IBM RISC System/6000, 1990): when q is within one ulp of a / d and
// r = a - d q is exact, q + r y rounds to the correctly rounded quotient.  The product a y is within two
// ulps; the first correction brings it within one, the second is the theorem's.  Asked for: quotients in the
// normal range, and remainders, multiples of about 2^-47 a, no finer than the smallest subnormal
// (division_in_range).  Zero numerators give zero.
PB_DIVIDE_FN float divide_by(float a, float d, float y) {
#ifdef __CUDA_ARCH__
    float q = __fmul_rn(a, y);
    q = __fmaf_rn(__fmaf_rn(-d, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-d, q, a), y, q);
#else
    float q = a * y;
    q = fmaf(fmaf(-d, q, a), y, q);
    return fmaf(fmaf(-d, q, a), y, q);
#endif
}

// Gradient sums are multiples of inv_scale below 2^44 inv_scale, so the squares divided here are zero or
// between inv_scale^2 / 2 and 2^88 inv_scale^2, the divisors between lambda and 2^13 + lambda.  At the ends
// of what is let through: quotients from 2^-122 to 2^98 (a row behind a square makes its divisor 1 at
// least), remainders multiples of 2^-145.
PB_DIVIDE_FN bool division_in_range(float inv_scale, float lam) {
    return inv_scale >= 3.5527137e-15f && inv_scale <= 32.f && lam >= 5.9604645e-8f && lam <= 16777216.f;  // 2^-48, 2^5; 2^-24, 2^24
}

}  // namespace pb
