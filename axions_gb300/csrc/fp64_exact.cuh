// Exact FP64 helpers of the FP64 step kernels: each returns the very double
// the plain IEEE operation would, with fewer instructions on the FP64 pipe
// (1/64 of the FP32 rate on GB300).  Only CUDA's IEEE intrinsics are used, so
// the results do not depend on the translation unit's -fmad setting.
#pragma once

#include <cuda_runtime.h>

namespace lat {

// x * p for an exact power of two p = 2^e.  When x and the result are normal
// numbers the product only moves the exponent field, which integer
// instructions do off the FP64 pipe (1/64 of the FP32 rate on GB300); zeros,
// subnormals, Inf/NaN and results outside the normal range take the FP64
// multiply.  Both give the same double.
__device__ __forceinline__ double mul_pow2(double x, double p)
{
    const long long bx = __double_as_longlong(x);
    const int ex = (int)(bx >> 52) & 0x7ff;
    const int e = ((int)(__double_as_longlong(p) >> 52) & 0x7ff) - 1023;
    const int ey = ex + e;
    if (ex == 0 || ex == 0x7ff || ey <= 0 || ey >= 0x7ff) return x * p;
    return __longlong_as_double(bx + ((long long)e << 52));
}

// The IEEE quotient a / b for a divisor b whose reciprocal y = RN(1/b) was
// computed on the host, by integer instructions: GB300 issues 2 FP64
// instructions per SM and cycle, and its integer pipes have time while an FP64
// step runs.  With the 53-bit mantissas A, B, Y of a, b, y, the high word of
// A*Y is A/B scaled, off by less than two units of the quotient's 53 bits
// (y's rounding); the remainder A*2^s - q*B, exact modulo 2^64, then tells
// which neighbour is nearest.  A quotient of two 53-bit numbers never lies
// halfway between two doubles.  (Before: the Markstein quotient on the FP64
// pipe, five instructions, 80 SM cycles a warp against about 25.)  |a| or |b|
// outside [2^-400, 2^401) (subnormals, Inf/NaN, and wherever the quotient
// could leave the normal range) take the IEEE division; a zero a returns +-0.
__device__ __forceinline__ double cdiv(double a, double b, double y)
{
    typedef unsigned long long u64;
    constexpr unsigned lo = 1023 - 400, span = 800;  // biased exponents lo .. lo + span
    const u64 ba = (u64)__double_as_longlong(a), bb = (u64)__double_as_longlong(b), by = (u64)__double_as_longlong(y);
    const unsigned ea = (unsigned)(ba >> 52) & 0x7ffu, eb = (unsigned)(bb >> 52) & 0x7ffu;
    const u64 sign = (ba ^ bb) & 0x8000000000000000ull;
    if (ea - lo > span || eb - lo > span) {
        if ((ba << 1) == 0 && eb - lo <= span) return __longlong_as_double((long long)sign);
        return a / b;
    }
    const u64 mask = 0xfffffffffffffull, one = 0x10000000000000ull;
    const u64 A = (ba & mask) | one, B = (bb & mask) | one, Y = (by & mask) | one;
    // A*Y*2^-42 = (A/B)*2^63, or 2^62 where B = 2^52 (then Y = 2^52 too)
    const u64 An = A << 11, Yn = Y << 11;
    const unsigned ah = (unsigned)(An >> 32), al = (unsigned)An, yh = (unsigned)(Yn >> 32), yl = (unsigned)Yn;
    const u64 H = (u64)ah * yh + (((u64)ah * yl) >> 32) + (((u64)al * yh) >> 32);
    const int below = A < B ? 1 : 0;                      // the quotient is A*2^(52 + below) / B
    const int shift = 11 - below - (B == one ? 1 : 0);
    u64 q = (H >> shift) + ((H >> (shift - 1)) & 1);
    const long long rem = (long long)((A << (52 + below)) - q * B);   // exact: |rem| < 2.6 B < 2^55
    const long long r2 = 2 * rem, m = (long long)B;
    q += (u64)((r2 > m ? 1 : 0) + (r2 > 3 * m ? 1 : 0) - (r2 < -m ? 1 : 0) - (r2 < -3 * m ? 1 : 0));
    return __longlong_as_double((long long)(sign | (((u64)(ea - eb + 1022u - (unsigned)below) << 52) + q)));
}

// The IEEE product a * b by integer instructions, for steps that the FP64 pipe
// bounds: the 53-bit mantissas' exact 106-bit product, rounded to nearest even.
// A product costs the integer pipes about as long as the FP64 pipe (some 30
// instructions), but the two run side by side.  Operands that enter several
// products are unpacked once.  Both factors have to be in product_range,
// [2^-510, 2^512): no zeros, subnormals, Inf or NaN, and no product that leaves
// the normal range.
struct Factor {
    unsigned long long m;   // the mantissa, its leading one at bit 63
    unsigned hi;            // the high word: sign and exponent
};

__device__ __forceinline__ Factor factor(double a)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(a);
    return Factor{(b << 11) | 0x8000000000000000ull, (unsigned)(b >> 32)};
}

// 0 .. kProductSpan-1 exactly for a double in product_range; the maximum over
// several values tells whether all are
constexpr unsigned kProductSpan = 1022u << 20;   // biased exponents 513 .. 1534
__device__ __forceinline__ unsigned product_range(double a)
{
    return ((unsigned)((unsigned long long)__double_as_longlong(a) >> 32) & 0x7fffffffu) - (513u << 20);
}

__device__ __forceinline__ double mul(const Factor& a, const Factor& b)
{
    typedef unsigned long long u64;
    const unsigned ah = (unsigned)(a.m >> 32), al = (unsigned)a.m, bh = (unsigned)(b.m >> 32), bl = (unsigned)b.m;
    const u64 t0 = (u64)al * bl, t1 = (u64)ah * bl + (t0 >> 32), t2 = (u64)al * bh + (unsigned)t1;
    u64 h = (u64)ah * bh + (t1 >> 32) + (t2 >> 32);   // in [2^62, 2^64); below it (t2, t0) low words
    // The product's lowest 22 bits are zero, so the top bit of the low half and
    // whether anything is left of it are in t2's low word and t0's.
    const int below = (int)(h >> 63) ^ 1;             // the product is under 2: one bit more
    const unsigned l2 = (unsigned)t2;
    h = (h << below) | (below ? l2 >> 31 : 0u);
    const unsigned rest = ((unsigned)h & 0x7ffu) | (((l2 << below) | (unsigned)t0) != 0 ? 1u : 0u);
    u64 n = h >> 11;
    // the bits below the last one: above half, or half and the last one odd
    n += (rest + ((unsigned)n & 1u)) > 0x400u ? 1 : 0;
    const unsigned e = ((a.hi & 0x7ff00000u) + (b.hi & 0x7ff00000u)) - ((1023u + (unsigned)below) << 20);
    return __longlong_as_double((long long)(n + ((u64)(e + ((a.hi ^ b.hi) & 0x80000000u)) << 32)));
}

// The same where a may also be zero (the sine of a vanishing angle)
__device__ __forceinline__ unsigned product_range_or_zero(double a)
{
    return (__double_as_longlong(a) << 1) == 0 ? 0 : product_range(a);
}
__device__ __forceinline__ double mul_or_zero(double a, double b)
{
    const unsigned long long sign =
        (unsigned long long)(__double_as_longlong(a) ^ __double_as_longlong(b)) & 0x8000000000000000ull;
    const double r = mul(factor(a), factor(b));
    return (__double_as_longlong(a) << 1) == 0 ? __longlong_as_double((long long)sign) : r;
}

}  // namespace lat
