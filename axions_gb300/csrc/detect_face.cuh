// One face of the bilinear string detection (detect.cu): its roots in the
// reference's double-precision arithmetic, and the FP32 test that proves most
// faces to have none.  Compiled with -fmad=false.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace lat {

struct Roots {
    int n;
    double s1[2], s2[2];
};

// One face: v00 at (u,w), v10 at (u+du,w), v01 at (u,w+dw), v11 at (u+du,w+dw).
__device__ __forceinline__ Roots face_roots(const double v00[2], const double v10[2], const double v01[2],
                                            const double v11[2], double u, double w, double du, double dw)
{
    double coeff1[2], coeff2[2], coeff3[2], coeff4[2];
#pragma unroll
    for (int comp = 0; comp < 2; ++comp) {
        coeff1[comp] = v11[comp] - v10[comp] - v01[comp] + v00[comp];
        coeff2[comp] = (w + dw) * (v10[comp] - v00[comp]) + w * (v01[comp] - v11[comp]);
        coeff3[comp] = (u + du) * (v01[comp] - v00[comp]) + u * (v10[comp] - v11[comp]);
        coeff4[comp] = (u + du) * ((w + dw) * v00[comp] - w * v01[comp]) - u * ((w + dw) * v10[comp] - w * v11[comp]);
    }
    const double a = coeff1[1] * coeff3[0] - coeff1[0] * coeff3[1];
    const double b = coeff1[1] * coeff4[0] + coeff2[1] * coeff3[0] - coeff1[0] * coeff4[1] - coeff2[0] * coeff3[1];
    const double c = coeff2[1] * coeff4[0] - coeff2[0] * coeff4[1];
    const double discrim = b * b - 4 * a * c;
    Roots r;
    r.n = 0;
    if (a == 0) {
        if (b != 0) {
            const double sol2 = -c / b;
            if (sol2 >= w && sol2 <= w + dw) {
                const double sol1 = -(coeff3[0] * sol2 + coeff4[0]) / (coeff1[0] * sol2 + coeff2[0]);
                if (sol1 >= u && sol1 <= u + du) { r.s1[r.n] = sol1; r.s2[r.n] = sol2; r.n++; }
            }
        }
    } else if (discrim >= 0) {
        const double sq = sqrt(discrim);
        double sol2 = (-b + sq) / (2 * a);
        if (sol2 >= w && sol2 <= w + dw) {
            const double sol1 = -(coeff3[0] * sol2 + coeff4[0]) / (coeff1[0] * sol2 + coeff2[0]);
            if (sol1 >= u && sol1 <= u + du) { r.s1[r.n] = sol1; r.s2[r.n] = sol2; r.n++; }
        }
        sol2 = (-b - sq) / (2 * a);
        if (sol2 >= w && sol2 <= w + dw) {
            const double sol1 = -(coeff3[0] * sol2 + coeff4[0]) / (coeff1[0] * sol2 + coeff2[0]);
            if (sol1 >= u && sol1 <= u + du) { r.s1[r.n] = sol1; r.s2[r.n] = sol2; r.n++; }
        }
    }
    return r;
}

// ---- which faces can hold a crossing -----------------------------------------
// face_roots costs some 100 FP64 instructions a face, and GB300 issues only 2
// per SM and cycle: evaluated on every face, a count took 10.7 ms on 256^3.
// Most faces hold no crossing by a wide margin, which FP32 arithmetic (1/64 of
// the cost) on the corner values can prove; only the others, packed so that
// no lane idles, go through face_roots.  With s, t in [0, 1] along u, w and
//   v_c(s, t) = A_c + B_c s + C_c t + D_c s t     (c = 0, 1),
// face_roots solves q(t) = a t^2 + b t + e = 0, the resultant of v_0 and v_1,
// for t = (sol2 - w)/dw and takes s from v_0 = 0.  Three proofs that it returns
// no root, after scaling the corners by a power of two to max|v| in [1, 2):
//  1. v_0 has one sign at the corners, beyond `kappa`: sol1 is computed from
//     v_0 = 0, so v_0 at an accepted point is zero to rounding, yet it lies
//     between the corner values there.
//  2. q's discriminant is negative beyond its error.
//  3. Both roots of q are known well enough (a and the discriminant clear of
//     their errors) and each is outside [0, 1], or v_0 has one sign on the
//     line t = const for every t within the root's error.
// Errors: E bounds what q(t) is off for 0 <= t <= 1, here (corners truncated to
// 24 bits: 2^-18 and 2^-20 per unit of the differences) and in face_roots,
// which works in lattice coordinates up to N = n/2 spacings from the origin,
// where the terms of the resultant reach N^3 times its own size: 16 eps N^3,
// passed as `eref`.  A root is then off by at most 8 E / sqrt(discriminant);
// textbook roots, as face_roots forms them, add eps N (1 + |b/a|), which the
// bound on a covers.  Corners outside the FP32 range, NaN and Inf are never
// rejected (the comparisons fail).
__device__ __forceinline__ float corner_float(float v) { return v; }
__device__ __forceinline__ float corner_float(double v)
{
    // v truncated to 24 bits by integer instructions (a conversion takes the
    // FP64 pipe); below the float range 0, above it Inf
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v), m = hi & 0x7fffffffu;
    unsigned f = ((m - (896u << 20)) << 3) | (lo >> 29);
    f = m < (897u << 20) ? 0u : (m >= (1151u << 20) ? 0x7f800000u : f);
    return __uint_as_float(f | (hi & 0x80000000u));
}

struct Corner {
    float x, y;  // components 0 and 1
};

__device__ __forceinline__ bool face_maybe(const Corner& p00, const Corner& p10, const Corner& p01, const Corner& p11,
                                           float eref)
{
    const float m0 = fmaxf(fmaxf(fabsf(p00.x), fabsf(p10.x)), fmaxf(fabsf(p01.x), fabsf(p11.x)));
    const float lo0 = fminf(fminf(p00.x, p10.x), fminf(p01.x, p11.x));
    const float hi0 = fmaxf(fmaxf(p00.x, p10.x), fmaxf(p01.x, p11.x));
    const float kappa = (0x1p-12f + eref) * m0;
    const float sum = ((p00.x + p10.x) + (p01.x + p11.x)) + ((p00.y + p10.y) + (p01.y + p11.y));
    if (!(fabsf(sum) < 1e37f)) return true;                 // NaN, Inf or out of range
    if (m0 > 0x1p-100f && (lo0 > kappa || hi0 < -kappa)) return false;                                  // 1
    const float m1 = fmaxf(fmaxf(fabsf(p00.y), fabsf(p10.y)), fmaxf(fabsf(p01.y), fabsf(p11.y)));
    const float m = fmaxf(m0, m1);
    if (!(m > 0x1p-100f && m < 0x1p100f)) return true;
    const float sc = __uint_as_float((254u << 23) - (__float_as_uint(m) & 0x7f800000u));   // 2^-exponent(m)
    const float A0 = p00.x * sc, A1 = p00.y * sc;
    const float B0 = p10.x * sc - A0, B1 = p10.y * sc - A1;
    const float C0 = p01.x * sc - A0, C1 = p01.y * sc - A1;
    const float D0 = (p11.x - p10.x) * sc - C0, D1 = (p11.y - p10.y) * sc - C1;
    const float a = C1 * D0 - C0 * D1;
    const float b = A1 * D0 + C1 * B0 - A0 * D1 - C0 * B1;
    const float e = A1 * B0 - A0 * B1;
    const float E = 0x1p-18f + 0x1p-20f * (fabsf(B0) + fabsf(B1) + fabsf(C0) + fabsf(C1) + fabsf(D0) + fabsf(D1)) + eref;
    const float disc = b * b - 4.f * a * e;
    const float edisc = 4.f * E * (fabsf(a) + fabsf(b) + fabsf(e)) + 8.f * E * E;
    if (disc < -2.f * edisc) return false;                                                              // 2
    const float sq = sqrtf(fmaxf(disc, 0.f));
    if (!(fabsf(a) >= 8.f * E && sq >= 256.f * E && disc > 2.f * edisc)) return true;
    const float h = -0.5f * (b + (b < 0.f ? -sq : sq));     // the roots h/a and e/h, neither cancels
    const float dt = 8.f * E / sq;
    const float eta = (fabsf(C0) + fabsf(D0)) * dt + E + 0x1p-18f;
    bool maybe = false;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float t = r ? e / h : h / a;
        if (t < -dt || t > 1.f + dt) continue;
        const float v_s0 = A0 + C0 * t, v_s1 = v_s0 + B0 + D0 * t;
        if ((v_s0 > eta && v_s1 > eta) || (v_s0 < -eta && v_s1 < -eta)) continue;
        maybe = true;                                                                                   // not 3
    }
    return maybe;
}

}  // namespace lat
