// Quotients by constants without a division, equal to the IEEE quotient after rounding to the 16-bit type.  Plain C++ so
// that the host can run every one of the 65 536 inputs through the very function the kernels use (tests/test_exact_div.py).
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define FQ_HD __host__ __device__ __forceinline__
#else
#define FQ_HD inline
#endif

namespace fq {

// d / top for a 16-bit value d >= 0 and top = 15 or 255, rtop = fp32(1 / top): the product with the rounded reciprocal and one
// residual step (Markstein, IBM J. Res. Dev. 34, 1990).  Rounded to d's type it equals the rounded IEEE quotient for every
// finite d; an infinity or a NaN would leave the residual step as a NaN and is its own quotient.
FQ_HD float div_by_top(float d, float top, float rtop) {
    const float q0 = d * rtop;
    const float q = fmaf(fmaf(-q0, top, d), rtop, q0);
    return d <= 3.402823466e38f ? q : d;
}

// x / fp32(sqrt(128)) rounded to x's 16-bit type equals x * TURBO_RCD so rounded, TURBO_RCD two ulps above fp32(1 / sqrt(128)).
constexpr float TURBO_RCD = 0.0883883610367775f;

}  // namespace fq
