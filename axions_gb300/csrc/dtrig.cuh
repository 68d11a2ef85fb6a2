// Double-precision sine and cosine for the FP64 step kernels, evaluated on
// the integer pipe.
//
// GB300 issues FP64 at 2 instructions per SM and cycle, integer at 64 or
// more: one FP64 instruction costs the FP64 pipe as much as 32 integer ones
// cost theirs, and the two pipes run side by side.  So of a sine or cosine
// only the subtraction that reduces the argument stays in FP64 (two
// instructions); the rest is fixed-point arithmetic on 64-bit integers:
//
//   x = k*pi/2 + r, |r| <= pi/4(1 + 2^-6): k from a float copy of x (FP32),
//       r by a two-part Cody-Waite step (Cody & Waite 1980): k*P1 is exact
//       (16 + 36 bits), the second FMA rounds once;
//   r = m*2^e with m in [1/2, 1) as a 64-bit fraction, z = r^2 likewise;
//   sin r = r*S(z), cos r = C(z): the Taylor polynomials of degree 9 in z
//       (truncation below 2^-66) by Horner's rule, the first steps on 32-bit
//       words (their terms are below 2^-24), the others on 64-bit ones.
//       r*S(z) is formed on the normalised m, so a sine near a zero keeps its
//       relative accuracy;
//   the 64-bit result is rounded to the double.
//
// At most 1.65 ulps: the rounding of r is half a unit of r, a whole one of a result
// just below a power of two, pi/2's 2^-92.8 up to 0.09 and the integers 0.06 of one,
// and the final rounding is half of one.  Over 750,000 samples at multiples of pi/2
// and of pi/4 and powers of two from them 1.49 was found, over random ones 1.35
// (mean 0.29).  CUDA documents 2 ulps for its double sin.
// Measured on GB300, SM cycles for a warp's evaluation: sine 65, sincos 95.
// The table-driven form before it, all on the FP64 pipe (13 and 15
// instructions, at most 2.45 ulps), took 234 and 266.
//
// Only integer operations and explicit IEEE intrinsics are used, so the
// results do not depend on the translation unit's -fmad setting: the strict
// and fast FP64 kernels and the one-pass kernel get the very same doubles.
//
// |x| >= 2^16 (where k no longer fits the exact product), NaN/Inf and arguments
// within 2^-20 of a multiple of pi/2 other than 0 go to CUDA's sin/cos; |x| < 2^-27 returns sin x = x, cos x = 1.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

namespace lat {

namespace dtrig {

constexpr int kHiLarge = 0x40f00000;  // high word of 2^16
constexpr int kHiTiny = 0x3e400000;   // high word of 2^-27

// pi/2 = P1 + P2 within 2^-92.8: 36 bits, then the nearest double of the rest
constexpr double kP1 = 0x1.921fb54440000p+0;
constexpr double kP2 = 0x1.68c234c4c6629p-39;

// Taylor coefficients 1/(2n+1)! and 1/(2n)!: n = 0..5 as fractions of 2^64
// (1 as 2^64 - 1), n = 6..9 as fractions of 2^60
constexpr uint64_t kOne = 0xffffffffffffffffull;
constexpr uint64_t kS1 = 0x2aaaaaaaaaaaaaabull, kS2 = 0x0222222222222222ull,
                   kS3 = 0x000d00d00d00d00dull, kS4 = 0x00002e3bc74aad8eull, kS5 = 0x0000006b99159fd5ull;
constexpr uint32_t kS6 = 0x0b09230au, kS7 = 0x000d73fau, kS8 = 0x00000ca9u, kS9 = 0x00000009u;
constexpr uint64_t kC1 = 0x8000000000000000ull, kC2 = 0x0aaaaaaaaaaaaaabull,
                   kC3 = 0x005b05b05b05b05bull, kC4 = 0x0001a01a01a01a02ull, kC5 = 0x0000049f93edde28ull;
constexpr uint32_t kC6 = 0x8f76c780u, kC7 = 0x00c9cba5u, kC8 = 0x0000d740u, kC9 = 0x000000b4u;

__device__ __forceinline__ uint32_t float_bits(float f)
{
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
__device__ __forceinline__ float bits_float(uint32_t u)
{
    float f;
    memcpy(&f, &u, 4);
    return f;
}
__device__ __forceinline__ uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// the high 64 bits of a*b, at most 3 too small (the low words' product is left out)
__device__ __forceinline__ uint64_t mul_hi(uint64_t a, uint64_t b)
{
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (uint64_t)ah * bh + mul_hi(ah, bl) + mul_hi(al, bh);
}

// r = x - k*pi/2 and k (its low bits) for 2^-27 <= |x| < 2^16.  The float
// copy of x is x truncated to 24 bits, moved there by integer instructions.
// `cancelled`: x is within 2^-20 of a multiple of pi/2 other than 0, where the
// second part of pi/2 no longer gives r to 53 bits.  (A third FMA there is
// compiled without a branch, so every call paid for it.)
__device__ __forceinline__ double reduce(double x, uint32_t& quadrant, bool& cancelled)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const uint32_t sign = hi & 0x80000000u;
    const float xf = bits_float(sign | ((((hi & 0x7fffffffu) - (896u << 20)) << 3) | (lo >> 29)));
    const float t = fmaf(xf, 0.636619772367581343f, 12582912.0f);  // 1.5*2^23: rounds to an integer
    quadrant = float_bits(t);
    const uint32_t kf = float_bits(t - 12582912.0f);
    const uint32_t ka = kf & 0x7fffffffu;
    // k as a double (at most 17 bits: the low word is zero)
    const uint32_t kh = (ka == 0 ? 0u : (ka >> 3) + (896u << 20)) | (kf & 0x80000000u);
    const double k = __longlong_as_double((long long)((uint64_t)kh << 32));
    const double r = __fma_rn(-k, kP2, __fma_rn(-k, kP1, x));
    cancelled = ka != 0 && ((uint32_t)__double2hiint(r) & 0x7fffffffu) < 0x3eb00000u;
    return r;
}

// |r| = m*2^(e - 1022) with m a fraction of 2^64 in [1/2, 1), and r^2
struct Arg {
    uint64_t m, z;
    int e;          // biased exponent of r
    uint32_t sign;  // the sign bit of r
};

__device__ __forceinline__ Arg arg_of(double r)
{
    const uint64_t b = (uint64_t)__double_as_longlong(r);
    Arg a;
    a.sign = (uint32_t)(b >> 32) & 0x80000000u;
    a.e = (int)(b >> 52) & 0x7ff;
    a.m = (b << 11) | 0x8000000000000000ull;
    const int s = 2 * (1022 - a.e);
    a.z = mul_hi(a.m, a.m) >> (s < 63 ? s : 63);
    return a;
}

// S(z), or C(z) where `odd`, as a fraction of 2^64.  One evaluation with the
// coefficients selected: a branch per quadrant would run both polynomials in
// a warp of mixed quadrants (88 SM cycles a warp's sine against 65).
__device__ __forceinline__ uint64_t poly(uint64_t z, bool odd)
{
    const uint32_t zh = (uint32_t)(z >> 32);
    uint32_t w = (odd ? kC8 : kS8) - mul_hi(zh, odd ? kC9 : kS9);
    w = (odd ? kC7 : kS7) - mul_hi(zh, w);
    w = (odd ? kC6 : kS6) - mul_hi(zh, w);
    uint64_t p = (odd ? kC5 : kS5) - (((uint64_t)zh * w) >> 28);
    p = (odd ? kC4 : kS4) - mul_hi(z, p);
    p = (odd ? kC3 : kS3) - mul_hi(z, p);
    p = (odd ? kC2 : kS2) - mul_hi(z, p);
    p = (odd ? kC1 : kS1) - mul_hi(z, p);
    return kOne - mul_hi(z, p);
}

// the double nearest to p*2^-64 * 2^(e - 1022), p >= 2^63
__device__ __forceinline__ uint64_t round_bits(uint64_t p, int e)
{
    return ((uint64_t)(uint32_t)(e - 1) << 52) + (p >> 11) + ((p >> 10) & 1);
}

// |sin r| (p = S(z)) and cos r (p = C(z)) as bits
__device__ __forceinline__ uint64_t sin_bits(const Arg& a, uint64_t p)
{
    p = mul_hi(a.m, p);
    const int up = (int)(p >> 63) ^ 1;
    return round_bits(p << up, a.e - up);
}
__device__ __forceinline__ uint64_t cos_bits(uint64_t p) { return round_bits(p, 1022); }

__device__ __forceinline__ double with_sign(uint64_t bits, uint32_t sign)
{
    return __longlong_as_double((long long)(bits | ((uint64_t)sign << 32)));
}

}  // namespace dtrig

__device__ __forceinline__ double dsin(double x)
{
    using namespace dtrig;
    const int hi = __double2hiint(x) & 0x7fffffff;
    uint32_t q;
    bool cancelled;
    const Arg a = arg_of(reduce(x, q, cancelled));
    if (hi >= kHiLarge || (cancelled && hi >= kHiTiny)) return ::sin(x);
    // quadrants 0..3: sin r, cos r, -sin r, -cos r
    const bool odd = q & 1;
    const uint64_t p = poly(a.z, odd);
    const uint64_t sb = sin_bits(a, p), cb = cos_bits(p);
    const double s = with_sign(odd ? cb : sb, (odd ? 0u : a.sign) ^ ((q << 30) & 0x80000000u));
    return hi < kHiTiny ? x : s;
}

__device__ __forceinline__ void dsincos(double x, double* sp, double* cp)
{
    using namespace dtrig;
    const int hi = __double2hiint(x) & 0x7fffffff;
    uint32_t q;
    bool cancelled;
    const Arg a = arg_of(reduce(x, q, cancelled));
    if (hi >= kHiLarge || (cancelled && hi >= kHiTiny)) {
        ::sincos(x, sp, cp);
        return;
    }
    const uint64_t sb = sin_bits(a, poly(a.z, false)), cb = cos_bits(poly(a.z, true));
    const bool odd = q & 1;
    const uint32_t ss = odd ? 0u : a.sign, cs = odd ? a.sign : 0u;
    const double s = with_sign(odd ? cb : sb, ss ^ ((q << 30) & 0x80000000u));
    const double c = with_sign(odd ? sb : cb, cs ^ (((q + 1) << 30) & 0x80000000u));
    *sp = hi < kHiTiny ? x : s;
    *cp = hi < kHiTiny ? 1.0 : c;
}

}  // namespace lat
