// The covariant Laplacian and the gauge current of the fused FP64 Abelian-Higgs
// update by 64-bit integer instructions.
//
// They take 38 of the 71 FP64 instructions of a site, on a pipe that issues 2 an
// SM and cycle and bounds the update.  As integers, a product of two mantissas is
// three 32 x 32-bit multiplications and a sum one addition after a shift, on pipes
// 32 times as wide.
//
// Every value keeps its own exponent, and every sum is aligned on the largest of
// its own terms, as a floating-point addition is: a product is truncated to 2^-59
// of itself, the sum of two of them to 2^-58 of the larger one, each of a Laplacian's
// seven terms to 2^-57 of the largest, where FP64 rounds each operation to 2^-53 of
// its result.  So a component, a neighbour, a site's scalar (at a string's core) or
// a sine that is small beside the others keeps the accuracy that FP64 gives it.
// (One exponent for all the values of a site, in units of 2^-60 of the largest,
// lost it: 2e-12 of the current where the scalar is 2^-20 of its neighbours.  It
// was no faster: 256^3 2113 us a plain step against 2085, 4427 and 4349 with
// diagnostics.)
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
// x >> n; 0, or the sign, for n >= 64
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
__host__ __device__ inline int64_t sar(int64_t x, unsigned n)
{
#ifdef __CUDA_ARCH__
    int64_t r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
    return r;
#else
    return x >> (n > 63 ? 63 : n);
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
__host__ __device__ inline unsigned larger(unsigned a, unsigned b) { return a > b ? a : b; }

// A link datum: the bits of its cosine or sine.
__host__ __device__ inline int64_t link_of(double v) { return (int64_t)bits_of(v); }
__host__ __device__ inline double link_value(int64_t q) { return of_bits((uint64_t)q); }

// A double as m * 2^(e - 1023 - 62), its sign in bit 31 of s: m in [2^62, 2^63),
// 0 for zero.  Subnormals, infinities and NaN are the caller's to leave out.
struct Num {
    uint64_t m;
    unsigned e, s;
};
__host__ __device__ inline Num num(uint64_t b)
{
    const unsigned h = (unsigned)(b >> 32);
    const uint64_t lead_bit = (uint64_t)((h & 0x7fffffffu) != 0 ? 0x40000000u : 0u) << 32;
    return Num{((b << 10) & 0x3fffffffffffffffull) | lead_bit, (h >> 20) & 0x7ffu, h};
}

// The high word of a * b, both below 2^63; at most 1 too small without EXACT
// (the low words' product left out).
template <bool EXACT = false>
__host__ __device__ inline uint64_t high(uint64_t a, uint64_t b)
{
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    uint64_t mid = (uint64_t)ah * bl + (uint64_t)al * bh;   // each below 2^63 - 2^32
    if constexpr (EXACT) mid += ((uint64_t)al * bl) >> 32;
    return (uint64_t)ah * bh + (mid >> 32);
}

// v * 2^(e - 2*1023 - 60)
struct Sum {
    int64_t v;
    unsigned e;
};
// t with the sign of bit 31 of s
__host__ __device__ inline int64_t with_sign(uint64_t t, unsigned s)
{
    const int64_t n = (int64_t)((int32_t)s >> 31);
    return ((int64_t)t ^ n) - n;
}
// a*b + c*d, flip1, flip2 = ~0: that product with the other sign.  |v| < 2^63, as
// each product is below 2^62
__host__ __device__ inline Sum dot(const Num& a, const Num& b, unsigned flip1, const Num& c, const Num& d, unsigned flip2)
{
    const unsigned e1 = a.e + b.e, e2 = c.e + d.e, e = larger(e1, e2);
    return Sum{with_sign(shr(high(a.m, b.m), e - e1), a.s ^ b.s ^ flip1) + with_sign(shr(high(c.m, d.m), e - e2), c.s ^ d.s ^ flip2), e};
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

// Exponents for which no result leaves the normal range: of the largest scalar; of
// any scalar or sine that is not zero (twice kLow is 60 bits above the least normal
// result); of a current that is not zero (three times biased).  (A product with a zero
// counts by its exponent too, which is under those of the others unless their sum is
// below 2^-950 of a neighbour.)
constexpr unsigned kTopLow = 560, kTopHigh = 1500, kLow = 548, kCurLow = 3 * 1023 - 940;

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
    // top: of the scalars; low: of what is not zero (x - 1 wraps to the largest
    // for zero); one: of the cosines, NaN and Inf above all others
    unsigned top = 0, low = ~0u, one = 0;
    auto magnitude = [](uint64_t b) { return (unsigned)(b >> 32) & 0x7fffffffu; };
    auto scalar = [&](double v) {
        const unsigned x = magnitude(bits_of(v));
        top = larger(top, x);
        low = x - 1 < low ? x - 1 : low;
    };
    auto link = [&](int64_t c, int64_t s) {
        const unsigned x = magnitude((uint64_t)s) - 1;
        one = larger(one, magnitude((uint64_t)c));
        low = x < low ? x : low;
    };
    scalar(p[0]), scalar(p[1]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        scalar(fwd[a][0]), scalar(fwd[a][1]), scalar(bwd[a][0]), scalar(bwd[a][1]);
        link(cs[a], sn[a]), link(csm[a], snm[a]);
    }
    if ((top >> 20) - kTopLow >= kTopHigh - kTopLow || low < (kLow << 20) - 1 || one >= 1024u << 20) return false;

    const Num p0 = num(bits_of(p[0])), p1 = num(bits_of(p[1]));
    // the site's scalar as a Sum: a cosine of 1 has exponent 1023, bit 62
    const Sum s0{with_sign(p0.m >> 2, p0.s), p0.e + 1023}, s1{with_sign(p1.m >> 2, p1.s), p1.e + 1023};
    Sum A[3], B[3], T0[3], T1[3];   // transported neighbours: forward, and the backward ones negated
    unsigned e0 = s0.e, e1 = s1.e;
    bool small = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const Num a0 = num(bits_of(fwd[a][0])), a1 = num(bits_of(fwd[a][1]));
        const Num c = num((uint64_t)cs[a]), s = num((uint64_t)sn[a]);
        A[a] = dot(a0, c, 0, a1, s, 0);
        B[a] = dot(a1, c, 0, a0, s, ~0u);
        const Num b0 = num(bits_of(bwd[a][0])), b1 = num(bits_of(bwd[a][1]));
        const Num cm = num((uint64_t)csm[a]), sm = num((uint64_t)snm[a]);
        T0[a] = dot(b1, sm, 0, b0, cm, ~0u);
        T1[a] = dot(b1, cm, ~0u, b0, sm, ~0u);
        e0 = larger(e0, larger(A[a].e, T0[a].e));
        e1 = larger(e1, larger(B[a].e, T1[a].e));

        const unsigned j1 = p1.e + A[a].e, j0 = p0.e + B[a].e, j = larger(j1, j0);
        // exact before the truncation: a uniform scalar's two products cancel
        auto times = [](const Num& x, const Sum& y, unsigned n) {
            const unsigned ys = (unsigned)((uint64_t)y.v >> 32);
            return with_sign(shr(high<true>((uint64_t)with_sign((uint64_t)y.v, ys), x.m), n), x.s ^ ys);
        };
        const int64_t q = times(p1, A[a], j - j1) - times(p0, B[a], j - j0);
        small |= q != 0 && j < kCurLow;
        cur[a] = to_double(q, (int)j - 3 * 1023 - 58);
        if constexpr (GRAD) {
            auto less = [&](const Sum& x, const Sum& t) {
                const unsigned e = larger(x.e, t.e);
                // |t.v| is up to 2^63; x.v has eight zero bits, and one bit stands for those that a longer shift leaves out
                const unsigned n = e - x.e + 1;
                const int64_t d = (sar(x.v, n) | (n > 8 ? 1 : 0)) + sar(t.v, e - t.e + 1);
                return to_double(d, (int)e - 2 * 1023 - 59);
            };
            grad[a][0] = less(s0, T0[a]);
            grad[a][1] = less(s1, T1[a]);
        }
    }
    // In eighths, which sum up to less than (6 * 2^63 + 6 * 2^61) / 8; the backward
    // terms subtracted, so that the truncations' means cancel.
    int64_t x0 = -sar(3 * s0.v, e0 - s0.e + 2), x1 = -sar(3 * s1.v, e1 - s1.e + 2);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        x0 += sar(A[a].v, e0 - A[a].e + 3) - sar(T0[a].v, e0 - T0[a].e + 3);
        x1 += sar(B[a].v, e1 - B[a].e + 3) - sar(T1[a].v, e1 - T1[a].e + 3);
    }
    u[0] = to_double(x0, (int)e0 - 2 * 1023 - 57);
    u[1] = to_double(x1, (int)e1 - 2 * 1023 - 57);
    return !small;
}

}  // namespace fix

}  // namespace lat
