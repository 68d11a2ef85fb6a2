// Abelian-Higgs FP64 step in two passes.
//
// FP64 on GB300 runs at 1/64 of the FP32 rate, so the step is bound by FP64
// instructions, not by HBM: the one-pass kernel (ah_step.cuh) evaluates every
// link's sin/cos and every plaquette sine twice, once for each site that
// needs it (as the reference does, mpi_evolution.cpp:418-487).  Here pass 1
// evaluates them once per site into a scratch buffer ("link data") and pass 2
// performs the update (mpi_evolution.cpp:412-501) reading the link data of the
// site and of its three backward neighbours.  The extra HBM traffic
// (~200 B/site) is small next to the FP64 time it saves.
//
// STRICT = true keeps the reference's rounding operation by operation (the
// translation unit is compiled with -fmad=false); the link data are the very
// doubles the one-pass kernel computes, so the two paths agree bit for bit.
// STRICT = false (LAT_F64_FAST) lets the compiler fuse multiply-adds and takes
// sin(P_yx) = -sin(P_xy) (likewise zx, zy): the same arithmetic to within an
// ulp per operation.
#pragma once

#include <type_traits>

#include "fixed_point.cuh"
#include "site_common.cuh"

namespace lat {

// link-data slots ([slot][N], SoA)
enum LinkSlot {
    L_CX, L_SX, L_CY, L_SY, L_CZ, L_SZ,   // cos/sin of theta_mu at the site
    L_PXY, L_PXZ, L_PYZ,                    // sin of P_xy, P_xz, P_yz at the site
    L_PYX, L_PZX, L_PZY,                    // sin of P_yx, P_zx, P_zy (STRICT only)
    L_CPXY, L_CPXZ, L_CPYZ,                 // cos of P_xy, P_xz, P_yz (diagnostic steps)
    L_COUNT
};

// Base address of every link-data slot.  The host forms them from the
// buffer and the site count in 64-bit arithmetic: an int slot*N + s offset
// would pass 2^31 above 143,165,576 sites (15 slots), where a kernel would
// write at a wrapped offset.  Inside one slot the site index s < 2^31.
template <class P>
struct LinkSlotsT {
    P p[L_COUNT];
};
using LinkSlots = LinkSlotsT<double* __restrict__>;
using LinkSlotsC = LinkSlotsT<const double* __restrict__>;

inline LinkSlots link_slots(double* L, long long N)
{
    LinkSlots s;
    for (int q = 0; q < L_COUNT; ++q) s.p[q] = L + (size_t)q * (size_t)N;
    return s;
}

inline LinkSlotsC link_slots_c(const double* L, long long N)
{
    LinkSlotsC s;
    for (int q = 0; q < L_COUNT; ++q) s.p[q] = L + (size_t)q * (size_t)N;
    return s;
}

// a / b where b = spacing^2 or spacing: the multiplication by the reciprocal,
// exact when every spacing is a power of two (then a*(1/b) == a/b for all a),
// else the IEEE quotient by cdiv from the host reciprocal.
template <bool RECIP>
__device__ __forceinline__ double sdiv(double a, double b, double inv_b)
{
    if constexpr (RECIP) return __dmul_rn(a, inv_b);
    else return cdiv(a, b, inv_b);
}

// x != 0 by integer instructions (a comparison of doubles takes the FP64 pipe)
__device__ __forceinline__ bool nonzero(double x) { return (__double_as_longlong(x) << 1) != 0; }

// t - a / b.  With power-of-two spacings the quotient is exact, so one fused
// operation rounds as the subtraction alone does.
template <bool RECIP>
__device__ __forceinline__ double sub_sdiv(double t, double a, double b, double inv_b)
{
    if constexpr (RECIP) return __fma_rn(-a, inv_b, t);
    else return t - cdiv(a, b, inv_b);
}

// x/dx2 + y/dy2 + z/dz2 - r, the quotients and sums rounded one by one (in that
// order); with power-of-two spacings the scalings are exact and fold into the
// additions, or, for equal spacings, into the last subtraction.
template <bool RECIP>
__device__ __forceinline__ double lap_minus(double x, double y, double z, double r, const StepCoef& c)
{
    if constexpr (RECIP) {
        if (nonzero(c.iso)) return __fma_rn(__dadd_rn(__dadd_rn(x, y), z), c.inv_dx2, -r);
        return __dadd_rn(__fma_rn(z, c.inv_dz2, __fma_rn(x, c.inv_dx2, __dmul_rn(y, c.inv_dy2))), -r);
    } else {
        return __dadd_rn(__dadd_rn(__dadd_rn(cdiv(x, c.dx2, c.inv_dx2), cdiv(y, c.dy2, c.inv_dy2)),
                                   cdiv(z, c.dz2, c.inv_dz2)), -r);
    }
}

// 2*x - y: the doubling is exact, so the fused form rounds once as the
// subtraction does
__device__ __forceinline__ double twice_minus(double x, double y) { return __fma_rn(2.0, x, -y); }
// t - 2*x
__device__ __forceinline__ double minus_twice(double t, double x) { return __fma_rn(-2.0, x, t); }

template <bool STRICT, bool DIAG>
__global__ void __launch_bounds__(BLOCK) ah_links_kernel(const Geom g, const Flat r, const double* __restrict__ TX,
                                                         const double* __restrict__ TY,
                                                         const double* __restrict__ TZ, const LinkSlots L)
{
    chain_wait();
    // g: the whole lattice as the region, so that q is the site index
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= r.n) return;
    const Nbr n = flat_nbr(g, r, q);
    const int s = n.s;
    const double tx = TX[s], ty = TY[s], tz = TZ[s];
    const double tyxp = TY[s + n.xp], tzxp = TZ[s + n.xp];
    const double txyp = TX[s + n.yp], tzyp = TZ[s + n.yp];
    const double txzp = TX[s + n.zp], tyzp = TY[s + n.zp];
    double sv, cv;
    dsincos(tx, &sv, &cv);
    L.p[L_CX][s] = cv;
    L.p[L_SX][s] = sv;
    dsincos(ty, &sv, &cv);
    L.p[L_CY][s] = cv;
    L.p[L_SY][s] = sv;
    dsincos(tz, &sv, &cv);
    L.p[L_CZ][s] = cv;
    L.p[L_SZ][s] = sv;
    // plaquette angles, summed in the reference's order (mpi_evolution.cpp:471-487)
    const double Pxy = tx + tyxp - txyp - ty;
    const double Pxz = tx + tzxp - txzp - tz;
    const double Pyz = ty + tzyp - tyzp - tz;
    if constexpr (DIAG) {
        dsincos(Pxy, &sv, &cv);
        L.p[L_PXY][s] = sv;
        L.p[L_CPXY][s] = cv;
        dsincos(Pxz, &sv, &cv);
        L.p[L_PXZ][s] = sv;
        L.p[L_CPXZ][s] = cv;
        dsincos(Pyz, &sv, &cv);
        L.p[L_PYZ][s] = sv;
        L.p[L_CPYZ][s] = cv;
    } else {
        L.p[L_PXY][s] = dsin(Pxy);
        L.p[L_PXZ][s] = dsin(Pxz);
        L.p[L_PYZ][s] = dsin(Pyz);
    }
    if constexpr (STRICT) {
        L.p[L_PYX][s] = dsin(ty + txyp - tyxp - tx);
        L.p[L_PZX][s] = dsin(tz + txzp - tzxp - tx);
        L.p[L_PZY][s] = dsin(tz + tyzp - tzyp - ty);
    }
}

// What the update of one site reads: the scalar and its neighbours, the past
// level, the link phases, and the link data of the site and of its backward
// neighbours (sP*_m: the plaquette sine there; sPyx, sPzx, sPzy in STRICT mode
// sines of their own, else the negated sPxy, sPxz, sPyz).
struct AhSite {
    double p0, p1, p0xp, p1xp, p0xm, p1xm, p0yp, p1yp, p0ym, p1ym, p0zp, p1zp, p0zm, p1zm;
    double q0, q1, tx, ty, tz, qx, qy, qz, txm, tym, tzm;
    double cx, sx, cy, sy, cz, sz, cxm, sxm, cym, sym, czm, szm;
    double sPxy, sPxz, sPyz, sPxy_m, sPxz_m, sPyz_m, sPyx, sPzx, sPzy, sPyx_m, sPzx_m, sPzy_m;
    double cPxy, cPxz, cPyz, divPast;   // diagnostic steps
};

// cm*x + sm*y, out of line: where a compiler would predicate it, it costs the
// FP64 pipe on every path
static __device__ __noinline__ double mul_add_rare(double cm, double x, double sm, double y)
{
    return __dadd_rn(__dmul_rn(cm, x), __dmul_rn(sm, y));
}

// How the strict update takes its products: on the FP64 pipe, or by integer
// instructions, with sines that may be zero or not (about 4 % slower if so).
// FIXED_POINT: the fused update of equal spacings, its Laplacian and current by
// fixed_point.cuh.
enum { FP_PRODUCTS, INT_PRODUCTS, INT_ZERO_SINES, FIXED_POINT };

// The update of one site (mpi_evolution.cpp:412-501) and its diagnostics: new
// values to `next` (phi, then theta), div(theta) to divNow.
template <bool STRICT, bool DIAG, bool RECIP, int INT>
__device__ __forceinline__ void ah_site(const AhSite& v, const StepCoef& c, const DiagOut& d, double (&next)[5],
                                        double& divNow, double& e_site, double& g_site)
{
    const double p0 = v.p0, p1 = v.p1, p0xp = v.p0xp, p1xp = v.p1xp, p0xm = v.p0xm, p1xm = v.p1xm;
    const double p0yp = v.p0yp, p1yp = v.p1yp, p0ym = v.p0ym, p1ym = v.p1ym;
    const double p0zp = v.p0zp, p1zp = v.p1zp, p0zm = v.p0zm, p1zm = v.p1zm;
    const double q0 = v.q0, q1 = v.q1, tx = v.tx, ty = v.ty, tz = v.tz, qx = v.qx, qy = v.qy, qz = v.qz;
    const double cx = v.cx, sx = v.sx, cy = v.cy, sy = v.sy, cz = v.cz, sz = v.sz;
    const double cxm = v.cxm, sxm_ = v.sxm, cym = v.cym, sym = v.sym, czm = v.czm, szm_ = v.szm;
    const double sPxy = v.sPxy, sPxz = v.sPxz, sPyz = v.sPyz, sPxy_m = v.sPxy_m, sPxz_m = v.sPxz_m, sPyz_m = v.sPyz_m;
    const double sPyx = v.sPyx, sPzx = v.sPzx, sPzy = v.sPzy;
    const double sPyx_m = v.sPyx_m, sPzx_m = v.sPzx_m, sPzy_m = v.sPzy_m;
    const double phiMagSqr = p0 * p0 + p1 * p1;
    const double pot = c.halfLambda * (phiMagSqr - c.etaSq);

    double tt0 = 0, tt1 = 0, curx, cury, curz;
    double gr[3][2];   // FIXED_POINT diagnostics: phi less its transported backward neighbours
    if constexpr (STRICT) {
        // INT: the products of the covariant Laplacian (mpi_evolution.cpp:418-428)
        // and of the current go through the integer pipes, where every factor
        // allows it: 42 of the update's 139 FP64 instructions.  With general
        // spacings the quotients take the integer pipes already, and the
        // current's outer products stay (128^3: 612 us a step, 635 without).
        // The remaining products, moved as well, gave nothing.
        const double val[20] = {p0,   p1,   p0xp, p1xp, p0yp, p1yp, p0zp, p1zp, p0xm, p1xm,
                                p0ym, p1ym, p0zm, p1zm, cx,   cy,   cz,   cxm,  cym,  czm};
        double br[6];
        const double sines[6] = {sx, sy, sz, sxm_, sym, szm_};
        unsigned range = INT != FP_PRODUCTS ? 0 : kProductSpan;
        if constexpr (INT != FP_PRODUCTS) {
#pragma unroll
            for (int k = 0; k < 20; ++k) range = max(range, product_range(val[k]));
#pragma unroll
            for (int k = 0; k < 6; ++k)
                range = max(range, INT == INT_ZERO_SINES ? product_range_or_zero(sines[k]) : product_range(sines[k]));
        }
        // times: a product; sine: one whose first factor is a sine
        auto terms = [&](auto times, auto sine) {
            // c = +1 then c = -1
            tt0 = lap_minus<RECIP>(minus_twice(times(cx, p0xp) + sine(sx, p1xp), p0) + times(cxm, p0xm) - sine(sxm_, p1xm),
                                   minus_twice(times(cy, p0yp) + sine(sy, p1yp), p0) + times(cym, p0ym) - sine(sym, p1ym),
                                   minus_twice(times(cz, p0zp) + sine(sz, p1zp), p0) + times(czm, p0zm) - sine(szm_, p1zm),
                                   pot * p0, c);
            tt1 = lap_minus<RECIP>(minus_twice(times(cx, p1xp) - sine(sx, p0xp), p1) + times(cxm, p1xm) + sine(sxm_, p0xm),
                                   minus_twice(times(cy, p1yp) - sine(sy, p0yp), p1) + times(cym, p1ym) + sine(sym, p0ym),
                                   minus_twice(times(cz, p1zp) - sine(sz, p0zp), p1) + times(czm, p1zm) + sine(szm_, p0zm),
                                   pot * p1, c);
            // brackets of the gauge current (mpi_evolution.cpp:459-466)
            br[0] = times(p1, p0xp) - times(p0, p1xp), br[1] = times(p0, p0xp) + times(p1, p1xp);
            br[2] = times(p1, p0yp) - times(p0, p1yp), br[3] = times(p0, p0yp) + times(p1, p1yp);
            br[4] = times(p1, p0zp) - times(p0, p1zp), br[5] = times(p0, p0zp) + times(p1, p1zp);
        };
        auto rounded = [](double x, double y) { return __dmul_rn(x, y); };
        bool in = INT != FP_PRODUCTS && range < kProductSpan;
        if (in) {
            auto sine = [](double x, double y) {
                if constexpr (INT == INT_ZERO_SINES) return mul_or_zero(x, y);
                else return mul(factor(x), factor(y));
            };
            terms([](double x, double y) { return mul(factor(x), factor(y)); }, sine);
            range = 0;
#pragma unroll
            for (int k = 0; k < 6; ++k) range = max(range, product_range(br[k]));
            in = RECIP && range < kProductSpan;
            if (in) {
                curx = mul(factor(cx), factor(br[0])) + sine(sx, br[1]);
                cury = mul(factor(cy), factor(br[2])) + sine(sy, br[3]);
                curz = mul(factor(cz), factor(br[4])) + sine(sz, br[5]);
            }
        } else {
            terms(rounded, rounded);
        }
        if (!in) {
            auto current = [](double cm, double x, double sm, double y) {
                if constexpr (INT != FP_PRODUCTS && RECIP) return mul_add_rare(cm, x, sm, y);
                else return __dadd_rn(__dmul_rn(cm, x), __dmul_rn(sm, y));
            };
            curx = current(cx, br[0], sx, br[1]);
            cury = current(cy, br[2], sy, br[3]);
            curz = current(cz, br[4], sz, br[5]);
        }
        if (nonzero(c.fric)) {
            tt0 = tt0 - c.fric * cdiv(p0 - q0, c.dt, c.inv_dt);
            tt1 = tt1 - c.fric * cdiv(p1 - q1, c.dt, c.inv_dt);
        }
    } else {
        // The same quantities with fewer FP64 instructions.  The forward
        // link-transported neighbour U_mu phi(x+mu), A = c phi0' + s phi1',
        // B = c phi1' - s phi0', enters both the Laplacian and the current:
        // j_mu = c (phi1 phi0' - phi0 phi1') + s (phi0 phi0' + phi1 phi1')
        //      = phi1 A - phi0 B.
        // FIXED_POINT: the sums less six times the scalar come from integers.
        double x0, x1, y0 = 0, y1 = 0, z0 = 0, z1 = 0;
        bool done = false;
        if constexpr (INT == FIXED_POINT) {
            using fix::link_of;
            const int64_t cs[3] = {link_of(cx), link_of(cy), link_of(cz)}, sn[3] = {link_of(sx), link_of(sy), link_of(sz)};
            const int64_t csm[3] = {link_of(cxm), link_of(cym), link_of(czm)};
            const int64_t snm[3] = {link_of(sxm_), link_of(sym), link_of(szm_)};
            double u[2], j[3];
            done = fix::scalar_terms<DIAG>({p0, p1}, {{p0xp, p1xp}, {p0yp, p1yp}, {p0zp, p1zp}},
                                     {{p0xm, p1xm}, {p0ym, p1ym}, {p0zm, p1zm}}, cs, sn, csm, snm, u, j, gr);
            x0 = u[0], x1 = u[1], curx = j[0], cury = j[1], curz = j[2];
        }
        if (!done) {
            auto direction = [&](double cp, double sp, double cm, double sm, double ap, double bp, double am, double bm,
                                 double& a, double& b, double& cur, double (&g)[2]) {
                const double A = fma(sp, bp, cp * ap), B = fma(-sp, ap, cp * bp);
                a = fma(-sm, bm, fma(cm, am, A)), b = fma(sm, am, fma(cm, bm, B));
                cur = fma(p1, A, -p0 * B);
                if constexpr (INT == FIXED_POINT && DIAG) {
                    g[0] = p0 - cm * am + sm * bm;
                    g[1] = p1 - cm * bm - sm * am;
                }
            };
            direction(cx, sx, cxm, sxm_, p0xp, p1xp, p0xm, p1xm, x0, x1, curx, gr[0]);
            direction(cy, sy, cym, sym, p0yp, p1yp, p0ym, p1ym, y0, y1, cury, gr[1]);
            direction(cz, sz, czm, szm_, p0zp, p1zp, p0zm, p1zm, z0, z1, curz, gr[2]);
            if constexpr (INT == FIXED_POINT) {
                x0 = fma(-6.0, p0, x0 + y0 + z0);
                x1 = fma(-6.0, p1, x1 + y1 + z1);
            }
        }
        if (INT == FIXED_POINT || nonzero(c.iso)) {
            // Equal spacings: every term of an update carries its factor dt^2
            // times a constant from the host and is added to the difference
            // of the two levels, which is small and exact, before that is
            // added to the level: 71 FP64 instructions a site, 33 with FIXED_POINT (74 with the
            // acceleration formed first) and one rounding of the level's size
            // instead of two.
            const double ps = c.kPot * (phiMagSqr - c.etaSq);
            const double s0 = INT == FIXED_POINT ? x0 : fma(-6.0, p0, x0 + y0 + z0);
            const double s1 = INT == FIXED_POINT ? x1 : fma(-6.0, p1, x1 + y1 + z1);
            const double u0 = fma(-ps, p0, s0), u1 = fma(-ps, p1, s1);
            double d0 = p0 - q0, d1 = p1 - q1, dx = tx - qx, dy = ty - qy, dz = tz - qz;
            if (nonzero(c.fric)) {
                d0 = fma(-c.kFric, d0, d0);
                d1 = fma(-c.kFric, d1, d1);
            }
            if (nonzero(c.damp)) {
                dx = fma(-c.kDamp, dx, dx);
                dy = fma(-c.kDamp, dy, dy);
                dz = fma(-c.kDamp, dz, dz);
            }
            next[0] = p0 + fma(c.kLap, u0, d0);
            next[1] = p1 + fma(c.kLap, u1, d1);
            // current and lattice curl (mpi_evolution.cpp:459-487)
            next[2] = tx + fma(c.kCur, curx, fma(-c.kLap, (sPxy - sPxy_m) + (sPxz - sPxz_m), dx));
            next[3] = ty + fma(c.kCur, cury, fma(-c.kLap, (sPyx - sPyx_m) + (sPyz - sPyz_m), dy));
            next[4] = tz + fma(c.kCur, curz, fma(-c.kLap, (sPzx - sPzx_m) + (sPzy - sPzy_m), dz));
        } else {
            tt0 = lap_minus<RECIP>(minus_twice(x0, p0), minus_twice(y0, p0), minus_twice(z0, p0), pot * p0, c);
            tt1 = lap_minus<RECIP>(minus_twice(x1, p1), minus_twice(y1, p1), minus_twice(z1, p1), pot * p1, c);
        }
    }

    if (STRICT || (INT != FIXED_POINT && !nonzero(c.iso))) {
        if constexpr (!STRICT) {
            if (nonzero(c.fric)) {
                tt0 = fma(-c.fric_dt, p0 - q0, tt0);
                tt1 = fma(-c.fric_dt, p1 - q1, tt1);
            }
        }

        // lattice curl (mpi_evolution.cpp:471-487)
        double ttx = sub_sdiv<RECIP>(c.m2gg * curx, sPxy - sPxy_m, c.dy2, c.inv_dy2);
        double tty = sub_sdiv<RECIP>(c.m2gg * cury, sPyx - sPyx_m, c.dx2, c.inv_dx2);
        double ttz = sub_sdiv<RECIP>(c.m2gg * curz, sPzx - sPzx_m, c.dx2, c.inv_dx2);
        ttx = sub_sdiv<RECIP>(ttx, sPxz - sPxz_m, c.dz2, c.inv_dz2);
        tty = sub_sdiv<RECIP>(tty, sPyz - sPyz_m, c.dz2, c.inv_dz2);
        ttz = sub_sdiv<RECIP>(ttz, sPzy - sPzy_m, c.dy2, c.inv_dy2);
        if (nonzero(c.damp)) {
            ttx = ttx - c.damp * cdiv(tx - qx, c.dt, c.inv_dt);
            tty = tty - c.damp * cdiv(ty - qy, c.dt, c.inv_dt);
            ttz = ttz - c.damp * cdiv(tz - qz, c.dt, c.inv_dt);
        }
        // mpi_evolution.cpp:432,499-501
        next[0] = twice_minus(p0, q0) + c.dt2 * tt0;
        next[1] = twice_minus(p1, q1) + c.dt2 * tt1;
        next[2] = twice_minus(tx, qx) + c.dt2 * ttx;
        next[3] = twice_minus(ty, qy) + c.dt2 * tty;
        next[4] = twice_minus(tz, qz) + c.dt2 * ttz;
    }

    divNow = 0;
    if (DIAG || d.store_div) {
        const double txm = v.txm, tym = v.tym, tzm = v.tzm;
        divNow = sdiv<RECIP>(tx - txm, c.dx2, c.inv_dx2) + sdiv<RECIP>(ty - tym, c.dy2, c.inv_dy2)
               + sdiv<RECIP>(tz - tzm, c.dz2, c.inv_dz2);
    }

    if constexpr (DIAG) {
        // energy density and Gauss deviation of the now level
        // (evolution.cpp:322-334,377-427; mpi_evolution.cpp:509-532).  Each
        // divisor other than dt occurs once per site, so cdiv's host
        // reciprocal replaces the division's own (the same doubles).
        const double cPxy = v.cPxy, cPxz = v.cPxz, cPyz = v.cPyz;
        const double pt0 = cdiv(p0 - q0, c.dt, c.inv_dt);
        const double pt1 = cdiv(p1 - q1, c.dt, c.inv_dt);
        if constexpr (INT != FIXED_POINT) {
            gr[0][0] = p0 - cxm * p0xm + sxm_ * p1xm;
            gr[0][1] = p1 - cxm * p1xm - sxm_ * p0xm;
            gr[1][0] = p0 - cym * p0ym + sym * p1ym;
            gr[1][1] = p1 - cym * p1ym - sym * p0ym;
            gr[2][0] = p0 - czm * p0zm + szm_ * p1zm;
            gr[2][1] = p1 - czm * p1zm - szm_ * p0zm;
        }
        const double px0 = sdiv<RECIP>(gr[0][0], c.dx, c.inv_dx), px1 = sdiv<RECIP>(gr[0][1], c.dx, c.inv_dx);
        const double py0 = sdiv<RECIP>(gr[1][0], c.dy, c.inv_dy), py1 = sdiv<RECIP>(gr[1][1], c.dy, c.inv_dy);
        const double pz0 = sdiv<RECIP>(gr[2][0], c.dz, c.inv_dz), pz1 = sdiv<RECIP>(gr[2][1], c.dz, c.inv_dz);
        double tdc = 0, fc = 0, gauss = 0;
        if (d.energy_form == LAT_ENERGY_MPI) {
            const double a0 = cdiv(tx - qx, c.dt, c.inv_dt), a1 = cdiv(ty - qy, c.dt, c.inv_dt),
                         a2 = cdiv(tz - qz, c.dt, c.inv_dt);
            tdc = 0.5 * (a0 * a0 + a1 * a1 + a2 * a2);
            fc = cdiv(1 - cPxy, c.gxy2, c.inv_gxy2) + cdiv(1 - cPxz, c.gxz2, c.inv_gxz2)
               + cdiv(1 - cPyz, c.gyz2, c.inv_gyz2);
        }
        if (nonzero(c.g)) {
            const double divPast = v.divPast;
            const double divThetat = cdiv(divNow - divPast, c.dt, c.inv_dt);
            gauss = cdiv(divThetat, c.g, c.inv_g) - c.twog * (p1 * pt0 - p0 * pt1);
            if (d.energy_form != LAT_ENERGY_MPI) {
                const double a0 = cdiv(tx - qx, c.gdtdx, c.inv_gdtdx), a1 = cdiv(ty - qy, c.gdtdy, c.inv_gdtdy),
                             a2 = cdiv(tz - qz, c.gdtdz, c.inv_gdtdz);
                tdc = 0.5 * (a0 * a0 + a1 * a1 + a2 * a2);
                const double Fxy = cdiv(1 - cPxy, c.gxy2, c.inv_gxy2);
                const double Fxz = cdiv(1 - cPxz, c.gxz2, c.inv_gxz2);
                const double Fyz = cdiv(1 - cPyz, c.gyz2, c.inv_gyz2);
                fc = Fxy + Fxz + Fyz;
            }
        }
        const double pm = phiMagSqr - c.etaSq;
        const double ed = pt0 * pt0 + pt1 * pt1 + px0 * px0 + px1 * px1 + py0 * py0 + py1 * py1 + pz0 * pz0
                        + pz1 * pz1 + tdc + fc + c.quarterLambda * (pm * pm);
        if (d.energy_form == LAT_ENERGY_MPI) e_site = ed * c.dx * c.dy * c.dz;
        else e_site = c.dV * ed;
        g_site = __longlong_as_double(__double_as_longlong(gauss) & 0x7fffffffffffffffll);
    }
}

// Lattices whose update moves FP64 work to integer instructions: those on which
// the FP64 pipe bounds it.  LAT_F64, us per step with FP64 products and with
// integer ones: 128^3 675 and 525 (diagnostic 1106 and 957; general spacings 665
// and 563), 64^3 96 and 77, 32^3 20.7 and 18.6 (diagnostic 40.8 and 38.6).  On
// smaller ones, with less than two warps for each scheduler, the longer chain of
// instructions counts: 24^3 diagnostic 31.5 and 33.6, general spacings 18.6 and
// 20.6.
// The fused form (equal spacings), FP64 and fixed_point.cuh: 256^3 3091 and 2085
// (diagnostic 5534 and 4349), 128^3 393 and 269, 64^3 54.6 and 40.2, 40^3 17.9
// and 15.2, 32^3 10.8 and 10.4, 24^3 8.2 and 9.0.
constexpr unsigned INT_SITES = 32 * 32 * 32;

// 128 registers: three blocks of 168 spill nothing and are no faster with plain
// steps (128^3: 527 us against 525), slower with diagnostic ones (1009 against 957).
constexpr int UPDATE_BLOCK = 128;   // flat_block's largest

template <bool STRICT, bool DIAG, bool RECIP, int INT>
__global__ void __launch_bounds__(UPDATE_BLOCK, 4)
ah_update_kernel(const Geom g, const Flat r, const Fields<double, 5> f, const LinkSlotsC L, const StepCoef c, const DiagOut d)
{
    chain_wait();
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    double e_site = 0.0, g_site = 0.0;

    if (q < r.n) {
        const Nbr n = flat_nbr(g, r, q);
        const int s = n.s;
        const int sxm = s + n.xm, sym = s + n.ym, szm = s + n.zm;
        const double* __restrict__ P0 = f.now[0];
        const double* __restrict__ P1 = f.now[1];
        AhSite v;
        v.p0 = P0[s], v.p1 = P1[s];
        v.p0xp = P0[s + n.xp], v.p1xp = P1[s + n.xp], v.p0xm = P0[sxm], v.p1xm = P1[sxm];
        v.p0yp = P0[s + n.yp], v.p1yp = P1[s + n.yp], v.p0ym = P0[sym], v.p1ym = P1[sym];
        v.p0zp = P0[s + n.zp], v.p1zp = P1[s + n.zp], v.p0zm = P0[szm], v.p1zm = P1[szm];
        v.q0 = f.past[0][s], v.q1 = f.past[1][s];
        v.tx = f.now[2][s], v.ty = f.now[3][s], v.tz = f.now[4][s];
        v.qx = f.past[2][s], v.qy = f.past[3][s], v.qz = f.past[4][s];
        v.cx = L.p[L_CX][s], v.sx = L.p[L_SX][s];
        v.cy = L.p[L_CY][s], v.sy = L.p[L_SY][s];
        v.cz = L.p[L_CZ][s], v.sz = L.p[L_SZ][s];
        v.cxm = L.p[L_CX][sxm], v.sxm = L.p[L_SX][sxm];
        v.cym = L.p[L_CY][sym], v.sym = L.p[L_SY][sym];
        v.czm = L.p[L_CZ][szm], v.szm = L.p[L_SZ][szm];
        v.sPxy = L.p[L_PXY][s], v.sPxz = L.p[L_PXZ][s], v.sPyz = L.p[L_PYZ][s];
        v.sPxy_m = L.p[L_PXY][sym], v.sPxz_m = L.p[L_PXZ][szm], v.sPyz_m = L.p[L_PYZ][szm];
        if constexpr (STRICT) {
            v.sPyx = L.p[L_PYX][s], v.sPzx = L.p[L_PZX][s], v.sPzy = L.p[L_PZY][s];
            v.sPyx_m = L.p[L_PYX][sxm], v.sPzx_m = L.p[L_PZX][sxm], v.sPzy_m = L.p[L_PZY][sym];
        } else {
            v.sPyx = -v.sPxy, v.sPzx = -v.sPxz, v.sPzy = -v.sPyz;
            v.sPyx_m = -L.p[L_PXY][sxm], v.sPzx_m = -L.p[L_PXZ][sxm], v.sPzy_m = -L.p[L_PYZ][sym];
        }
        if (DIAG || d.store_div) v.txm = f.now[2][sxm], v.tym = f.now[3][sym], v.tzm = f.now[4][szm];
        if constexpr (DIAG) {
            v.cPxy = L.p[L_CPXY][s], v.cPxz = L.p[L_CPXZ][s], v.cPyz = L.p[L_CPYZ][s];
            if (nonzero(c.g)) v.divPast = reinterpret_cast<const double*>(d.divbuf)[s];
        }
        double next[5], divNow;
        ah_site<STRICT, DIAG, RECIP, INT>(v, c, d, next, divNow, e_site, g_site);
        if (d.store_div) reinterpret_cast<double*>(d.divbuf)[s] = divNow;
        if (d.write) {  // in-place update of the past slot
#pragma unroll
            for (int m = 0; m < 5; ++m) f.past[m][s] = next[m];
        }
    }
    if constexpr (DIAG) flat_sum2_store(e_site, g_site, d.partials);
}

template <bool STRICT>
cudaError_t launch_ah_twopass(const Geom& g, const Fields<double, 5>& f, double* L, const StepCoef& c,
                              const DiagOut& d, bool diag, bool recip, cudaStream_t st)
{
    const long long N = (long long)g.nx * g.syz;
    const LinkSlots Lw = link_slots(L, N);
    const LinkSlotsC Lr = link_slots_c(L, N);
    Geom all = g;
    all.lox = all.loy = all.loz = 0;
    all.hix = g.nx;
    all.hiy = g.ny;
    all.hiz = g.nz;
    const Flat ra = flat_region(all);
    const int la = flat_grid(ra.n), lb = flat_block(ra.n);
    const Flat r = flat_region(g);
    const bool fixed = !STRICT && c.iso != 0 && r.n >= INT_SITES;
    cudaError_t e = launch_chained(diag ? ah_links_kernel<STRICT, true> : ah_links_kernel<STRICT, false>, la, lb, 0, st, all, ra,
                                   f.now[2], f.now[3], f.now[4], Lw);
    if (e != cudaSuccess) return e;
    const int grid = flat_grid(r.n), block = flat_block(r.n);
    auto go = [&](auto kernel) { e = launch_chained(kernel, grid, block, 0, st, g, r, f, Lr, c, d); };
    auto pick = [&](auto form) {
        constexpr int INT = decltype(form)::value;
        if (diag) recip ? go(ah_update_kernel<STRICT, true, true, INT>) : go(ah_update_kernel<STRICT, true, false, INT>);
        else recip ? go(ah_update_kernel<STRICT, false, true, INT>) : go(ah_update_kernel<STRICT, false, false, INT>);
    };
    if constexpr (STRICT) {
        if (r.n >= INT_SITES) {
            // the link phases vanish for good on fixed walls, and without coupling
            if (r.n != ra.n || c.g == 0) pick(std::integral_constant<int, INT_ZERO_SINES>{});
            else pick(std::integral_constant<int, INT_PRODUCTS>{});
            return e;
        }
    }
    if constexpr (!STRICT) {
        if (fixed) {
            pick(std::integral_constant<int, FIXED_POINT>{});
            return e;
        }
    }
    pick(std::integral_constant<int, FP_PRODUCTS>{});
    return e;
}

}  // namespace lat
