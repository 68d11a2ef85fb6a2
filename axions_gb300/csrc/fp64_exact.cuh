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

}  // namespace lat
