// Conversions and error-free arithmetic that stay off the FP64 pipe (which a
// conversion or a compare occupies as long as an FMA, 72 times an FP32 one).
#pragma once
#include <cuda_runtime.h>

namespace achr {
namespace {

// FP64 -> FP32 rounding toward zero with integer operations only.
// |v - f| <= 2^-23 |f| + 2^-126; tiny values flush to signed zero, overflow
// and inf map to inf.
__device__ __forceinline__ float f64_to_f32_rz(double v) {
    const unsigned hi = (unsigned)__double2hiint(v);
    const unsigned lo = (unsigned)__double2loint(v);
    const int fe = (int)((hi >> 20) & 0x7FFu) - 896;  // re-bias 1023 -> 127
    unsigned mag = ((unsigned)fe << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    mag = (fe <= 0) ? 0u : mag;
    mag = (fe >= 255) ? 0x7F800000u : mag;
    return __uint_as_float((hi & 0x80000000u) | mag);
}

// FP64 -> FP32 rounding to nearest (ties away from zero), otherwise like f64_to_f32_rz; not for NaN
// (its fraction's carry can reach the sign).
__device__ __forceinline__ float f64_to_f32_near(double v) {
    return f64_to_f32_rz(__longlong_as_double(__double_as_longlong(v) + (1ll << 28)));
}

// The same for any v, NaN giving an infinity: its exponent is looked at before the rounding.
__device__ __forceinline__ float f64_to_f32_near_any(double v) {
    const long long b = __double_as_longlong(v) + (1ll << 28);
    const unsigned hi = (unsigned)((unsigned long long)b >> 32), lo = (unsigned)b, was = (unsigned)__double2hiint(v);
    const int fe = (int)((hi >> 20) & 0x7FFu) - 896;
    unsigned mag = ((unsigned)fe << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    mag = (fe <= 0) ? 0u : mag;
    mag = (fe >= 255 || (was & 0x7FF00000u) == 0x7FF00000u) ? 0x7F800000u : mag;
    return __uint_as_float((was & 0x80000000u) | mag);
}

// Order-preserving integer key of a double (sign-magnitude -> two's
// complement; -0 and +0 share key 0).  a < b  <=>  key(a) < key(b) for non-NaN.
__device__ __forceinline__ long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    const long long mag = b & 0x7FFFFFFFFFFFFFFFll;
    return b < 0 ? -mag : mag;
}

// Exact clip of x to [lb, ub] (reference correctBounds, ACHRCuda.cu:198-202):
// x itself when inside, else the bound, compared through integer keys.
__device__ __forceinline__ double clip_exact(double x, double2 lu) {
    const long long kx = order_key(x);
    double r = x;
    if (kx < order_key(lu.x)) r = lu.x;
    if (kx > order_key(lu.y)) r = lu.y;
    return r;
}

// FP32 -> FP64 with integer operations only (exact for normal values; zero and
// subnormal values give a signed zero).
__device__ __forceinline__ double f32_to_f64_exact(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned e = (u >> 23) & 0xFFu;
    const unsigned long long s = (unsigned long long)(u & 0x80000000u) << 32;
    if (e == 0) return __longlong_as_double((long long)s);
    return __longlong_as_double(
        (long long)(s | ((unsigned long long)(e + 896u) << 52) | ((unsigned long long)(u & 0x7FFFFFu) << 29)));
}

// BF16 bits of f rounded to nearest even (hi) and of the remainder f - hi (lo),
// for finite f; FP32 and integer operations only.
__device__ __forceinline__ void split_bf16_bits(float f, unsigned short &hi, unsigned short &lo) {
    const unsigned u = __float_as_uint(f);
    const unsigned hu = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;
    hi = (unsigned short)(hu >> 16);
    const unsigned r = __float_as_uint(f - __uint_as_float(hu));
    const unsigned ru = (r + 0x7FFFu + ((r >> 16) & 1u)) & 0xFFFF0000u;
    lo = (unsigned short)(ru >> 16);
}

// High word of the smallest magnitude whose split is not that of the conversions, about 2^128 (1 - 2^-20):
// from there BF16 rounds to infinity, and an infinity or NaN comes out as an infinity and -0, or as 0.
constexpr unsigned kSplitTop = 0x47EFFFFFu;

// The split of such a value as the conversions give it: hi infinite and lo the opposite infinity; of an
// infinity hi infinite and lo NaN; of NaN both NaN.  A product with hi and lo is NaN.
__device__ __forceinline__ void split_bf16_top(double v, unsigned short &hi, unsigned short &lo) {
    const unsigned top = (unsigned)__double2hiint(v) & 0x7FFFFFFFu;
    const unsigned sign = ((unsigned)__double2hiint(v) >> 16) & 0x8000u;
    const bool finite = top < 0x7FF00000u, nan = !finite && (top > 0x7FF00000u || __double2loint(v) != 0);
    hi = (unsigned short)(nan ? 0x7FFFu : sign | 0x7F80u);
    lo = (unsigned short)(finite ? (sign ^ 0x8000u) | 0x7F80u : 0x7FFFu);
}

// Error-free transformations on FP32 (IEEE round-to-nearest; nvcc neither
// reassociates these nor contracts them beyond the explicit fmaf).
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float &s, float &e) {  // |a| >= |b| or a = 0
    s = __fadd_rn(a, b);
    e = __fsub_rn(b, __fsub_rn(s, a));
}
__device__ __forceinline__ void two_prod(float a, float b, float &p, float &e) {
    p = __fmul_rn(a, b);
    e = fmaf(a, b, -p);
}

// FP64 -> (hi, lo) FP32 with integer operations only: hi is v truncated to 24
// significant bits, lo the rest (up to 29 bits, rounded to 24); |v - hi - lo|
// <= 2^-48 |v|.  Values below 2^-126 become 0.
__device__ __forceinline__ void split_f64(double v, float &hi, float &lo) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7FF);
    const int fe = e - 896;  // FP32 biased exponent
    if (fe <= 0 || fe >= 255) {
        hi = (fe >= 255) ? __uint_as_float(sign | 0x7F800000u) : __uint_as_float(sign);
        lo = 0.0f;
        return;
    }
    const unsigned long long mant = b & 0xFFFFFFFFFFFFFull;
    hi = __uint_as_float(sign | ((unsigned)fe << 23) | (unsigned)(mant >> 29));
    const unsigned rest = (unsigned)(mant & 0x1FFFFFFFull);  // the low 29 bits: rest * 2^(e - 1075)
    const float r = __uint2float_rn(rest);
    const float l = ldexpf(r, e - 1075);
    lo = sign ? -l : l;
}

}  // namespace
}  // namespace achr
