// Correctly rounded FP64 quotient with integer and FP32 arithmetic (host and device).
//
// GB300's FP64 pipe takes 64 clocks for one instruction of a lone warp, so a
// compiled FP64 division (about nine dependent ones) costs 563 clocks there,
// and 140 clocks of the whole SM's FP64 pipe under load: for a 95-reaction
// chain, whose step is about 17 FP64 instructions besides, the two divisions
// of the ratio test were half the step.  This is schoolbook long division of
// the significands in three digits (21, 18 and 14 bits), each digit estimated
// as remainder x FP32 reciprocal of the divisor and corrected by the exact
// 64-bit remainder, and a rounding decided by the last remainder's sign.
#pragma once
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define ACHR_DIV_HD __host__ __device__ __forceinline__
#else
#define ACHR_DIV_HD inline
#endif

namespace achr {

ACHR_DIV_HD uint64_t div_bits(double v) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t b;
    memcpy(&b, &v, sizeof b);
    return b;
#endif
}
ACHR_DIV_HD double div_double(uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double v;
    memcpy(&v, &b, sizeof v);
    return v;
#endif
}
ACHR_DIV_HD float div_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float v;
    memcpy(&v, &b, sizeof v);
    return v;
#endif
}
ACHR_DIV_HD float div_rcp(float x) {  // relative error below 2^-21 suffices
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#elif defined(ACHR_DIV_RCP)  // (another one, for a test of the bound)
    return ACHR_DIV_RCP(x);
#else
    return 1.0f / x;
#endif
}

// a / b rounded to nearest even, for b > 0.  Positive normal a with a normal
// quotient takes the integer path; zero, negative, subnormal, infinite or NaN
// operands and quotients at the ends of the range are divided as usual.
ACHR_DIV_HD double div_rn(double a, double b) {
    const uint64_t ba = div_bits(a), bb = div_bits(b);
    const uint32_t ea = (uint32_t)(ba >> 52), eb = (uint32_t)(bb >> 52);  // sign and exponent
    const int e = (int)ea - (int)eb + 1023;
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || e < 2 || e > 2045) return a / b;
    const uint64_t one = 1ull << 52;
    uint64_t ma = (ba & (one - 1)) | one;
    const uint64_t mb = (bb & (one - 1)) | one;
    const int half = ma < mb ? 1 : 0;  // the quotient's significand lies in [1, 2)
    ma <<= half;
    // fb in [1, 2): mb / 2^52 truncated to 24 bits, r its reciprocal
    const float fb = div_float(0x3F800000u | (uint32_t)((mb >> 29) & 0x7FFFFFu));
    const float r = div_rcp(fb);
    // Digit 1: 2^21 ma / mb in [2^21, 2^22), off by at most 4.
    const float fa = (float)(int32_t)(ma >> 24);  // 2^-24 ma, below 2^30
    const int32_t q1 = (int32_t)(fa * (r * 0.0078125f));  // 2^(24 + 21 - 52) = 2^-7
    // Remainders are exact in 64-bit wrap-around arithmetic: |R1| <= 5 mb.
    const int64_t R1 = (int64_t)((ma << 21) - (uint64_t)(int64_t)q1 * mb);
    // Digit 2: 2^18 R1 / mb, below 2^21 in magnitude, off by at most 2.
    const int32_t q2 = (int32_t)((float)(int32_t)(R1 >> 26) * (r * 0.00390625f));  // 2^(26 + 18 - 52) = 2^-8
    const int64_t R2 = (int64_t)(((uint64_t)R1 << 18) - (uint64_t)(int64_t)q2 * mb);  // |R2| <= 2 mb
    // Digit 3: 2^14 R2 / mb, to nearest.
    const float f3 = (float)(int32_t)(R2 >> 26) * (r * 0.000244140625f);  // 2^(26 + 14 - 52) = 2^-12
    const int32_t q3 = (int32_t)(f3 + (f3 < 0.0f ? -0.5f : 0.5f));
    const int64_t R3 = (int64_t)(((uint64_t)R2 << 14) - (uint64_t)(int64_t)q3 * mb);  // |R3| < mb
    // 2^53 a/b = Q + R3 / mb.  The significand is Q / 2 to nearest; a tie cannot
    // occur (a quotient of two 53-bit numbers never ends in exactly half a unit).
    const uint64_t Q = (uint64_t)(((int64_t)q1 << 32) + ((int64_t)q2 << 14) + (int64_t)q3);
    const uint64_t m = (Q + (R3 > 0 ? 1u : 0u)) >> 1;
    return div_double(((uint64_t)(e - half) << 52) + (m - one));
}

}  // namespace achr
