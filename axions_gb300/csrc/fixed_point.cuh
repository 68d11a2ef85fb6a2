// The covariant Laplacian and the gauge current of the fused FP64 Abelian-Higgs
// update in 64-bit fixed point.
//
// They take 38 of the 71 FP64 instructions of a site, on a pipe that issues 2 an
// SM and cycle and bounds the update.  As integers, a product is a 64 x 64-bit
// multiplication's high word (about 9 instructions on pipes 32 times as wide)
// and a sum one addition.  The 14 scalar values that enter share the exponent of
// the largest (block floating point): units of 2^-60 of it, products truncated
// to 2^-58 of it, where FP64 rounds every product and sum to 2^-53 of its size.
// Link cosines and sines are multiples of 2^-62, exact for 1 and 0.
//
// Only integer operations: the host evaluates the same (for checks).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

namespace lat {

namespace fix {

__host__ __device__ inline uint64_t bits_of(double x)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
__host__ __device__ inline double of_bits(uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
// x >> n, 0 for n >= 64
__host__ __device__ inline uint64_t shr(uint64_t x, unsigned n)
{
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));   // clamps n at 64
    return r;
#else
    return n > 63 ? 0 : x >> n;
#endif
}
__host__ __device__ inline int64_t hi(int64_t a, int64_t b)
{
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}
__host__ __device__ inline unsigned lead(uint64_t x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__clzll((long long)x);
#else
    return (unsigned)__builtin_clzll(x);
#endif
}

__host__ __device__ inline unsigned exponent(uint64_t b) { return (unsigned)(b >> 52) & 0x7ffu; }

// The double with bits b, toward zero, in units of 2^(top - 1023 - 63 + drop),
// top no less than its exponent.  Zeros and subnormals give 0 (top > 64).
__host__ __device__ inline int64_t fixed(uint64_t b, unsigned top, unsigned drop)
{
    const uint64_t t = shr((b << 11) | 0x8000000000000000ull, top - exponent(b) + drop);
    const int64_t s = (int64_t)b >> 63;
    return ((int64_t)t ^ s) - s;
}

// x * 2^k to nearest even; the result has to be normal
__host__ __device__ inline double to_double(int64_t x, int k)
{
    const uint64_t sign = (uint64_t)x & 0x8000000000000000ull;
    uint64_t u = sign ? 0 - (uint64_t)x : (uint64_t)x;
    const unsigned n = lead(u | 1);
    u <<= n;
    uint64_t m = u >> 11;
    m += (((unsigned)u & 0x7ffu) + ((unsigned)m & 1u)) > 0x400u ? 1 : 0;
    m += (uint64_t)(unsigned)(k + 63 - (int)n + 1022) << 52;
    return of_bits(x == 0 ? 0 : (sign | m));
}

// a cosine or sine as a link datum: multiples of 2^-62, kNoLink for NaN
constexpr int64_t kNoLink = INT64_MIN;
__host__ __device__ inline int64_t link_of(double v)
{
    const uint64_t b = bits_of(v);
    return exponent(b) > 1023 ? kNoLink : fixed(b, 1023, 1);
}
__host__ __device__ inline double link_value(int64_t q) { return q == kNoLink ? of_bits(0x7ff8000000000000ull) : to_double(q, -62); }

// Exponents of the largest scalar for which every result is normal
constexpr unsigned kTopLow = 560, kTopHigh = 1500;

// u[comp]: the sum over the directions of the transported neighbours minus six
// times the site's scalar; cur[mu] = phi1 A_mu - phi0 B_mu, (A_mu, B_mu) the
// transported forward neighbour.  p: the site's scalar, fwd and bwd its
// neighbours', cs, sn, csm, snm the link data.  GRAD: grad[mu], the scalar less
// its transported backward neighbour.  false: out of range.
template <bool GRAD = false>
__host__ __device__ inline bool scalar_terms(const double (&p)[2], const double (&fwd)[3][2], const double (&bwd)[3][2],
                                             const int64_t (&cs)[3], const int64_t (&sn)[3], const int64_t (&csm)[3],
                                             const int64_t (&snm)[3], double (&u)[2], double (&cur)[3],
                                             double (*grad)[2] = nullptr)
{
    unsigned top = 0;
    int low = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const unsigned h = (unsigned)(bits_of(p[k]) >> 32) & 0x7fffffffu;
        top = top > h ? top : h;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const unsigned f = (unsigned)(bits_of(fwd[a][k]) >> 32) & 0x7fffffffu;
            const unsigned b = (unsigned)(bits_of(bwd[a][k]) >> 32) & 0x7fffffffu;
            top = top > f ? top : f;
            top = top > b ? top : b;
        }
        const int c0 = (int)(cs[a] >> 32), c1 = (int)(csm[a] >> 32);
        low = low < c0 ? low : c0;
        low = low < c1 ? low : c1;
    }
    top >>= 20;
    if (top - kTopLow >= kTopHigh - kTopLow || low < -(1 << 30)) return false;

    const int64_t f0 = fixed(bits_of(p[0]), top, 3), f1 = fixed(bits_of(p[1]), top, 3);   // below 2^61
    int64_t x0 = -((3 * f0) >> 1), x1 = -((3 * f1) >> 1);   // as the products: a quarter of the unit's count
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int64_t a0 = fixed(bits_of(fwd[a][0]), top, 3), a1 = fixed(bits_of(fwd[a][1]), top, 3);
        const int64_t b0 = fixed(bits_of(bwd[a][0]), top, 3), b1 = fixed(bits_of(bwd[a][1]), top, 3);
        const int64_t A = hi(a0, cs[a]) + hi(a1, sn[a]), B = hi(a1, cs[a]) - hi(a0, sn[a]);
        const int64_t t0 = hi(b0, csm[a]) - hi(b1, snm[a]), t1 = hi(b1, csm[a]) + hi(b0, snm[a]);
        x0 += A + t0;
        x1 += B + t1;
        if constexpr (GRAD) {
            grad[a][0] = to_double((f0 >> 2) - t0, (int)top - 1081);
            grad[a][1] = to_double((f1 >> 2) - t1, (int)top - 1081);
        }
        cur[a] = to_double(hi(f1, A * 4) - hi(f0, B * 4), 2 * (int)top - 2102);
    }
    u[0] = to_double(x0, (int)top - 1081);
    u[1] = to_double(x1, (int)top - 1081);
    return true;
}

}  // namespace fix

}  // namespace lat
