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

// Quotients d / sc of the code of an element, d >= 0 an fp32 number, rounded to the nearest integer (ties to even) like the IEEE
// quotient.  y: a reciprocal of sc within one ulp of it.
// After one residual step q differs from d / sc by less than 2^-45 of it.
//  * code_quotient16, sc of a 16-bit type (11 bits), codes up to 255: h * sc is an fp32 number for every half-integer h (20 bits),
//    so either d = h * sc, and the step gives h, or d is at least an ulp away, 2^-24 (1 + 2^-20) of it, and neither the IEEE
//    quotient nor q rounds to h: both lie on the same side.
//  * code_quotient32, any fp32 sc: the IEEE quotient itself.  refine_rcp rounds y correctly, one step brings q within an ulp, the
//    second to the quotient (Markstein, IBM J. Res. Dev. 34, 1990); but for a mantissa of sc of ones only, where refine_rcp gives a
//    NaN and the caller divides.
FQ_HD float code_quotient16(float d, float sc, float y) {
    const float q = d * y;
    return fmaf(fmaf(-q, sc, d), y, q);
}
FQ_HD float refine_rcp(float sc, float y) {
    union { float f; unsigned u; } b;
    b.f = sc;
    y = fmaf(fmaf(-sc, y, 1.0f), y, y);
    return (b.u & 0x7fffffu) == 0x7fffffu ? NAN : y;
}
FQ_HD float code_quotient32(float d, float sc, float y) {
    const float q = code_quotient16(d, sc, y);
    return fmaf(fmaf(-q, sc, d), y, q);
}

// x / fp32(sqrt(128)) rounded to x's 16-bit type equals x * TURBO_RCD so rounded, TURBO_RCD two ulps above fp32(1 / sqrt(128)).
constexpr float TURBO_RCD = 0.0883883610367775f;

}  // namespace fq
