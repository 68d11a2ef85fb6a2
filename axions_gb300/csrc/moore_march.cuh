// Moore-model FP64 leapfrog step marching along x: link data and update in one
// kernel.
//
// The one-pass kernel (moore_step.cuh) evaluates every link factor and plaquette
// sine for each site that uses it: 12 sincos and 12 sines a site, and more live
// values than fit the registers (1.34 ms on 96^3, 7,400 SM cycles a warp).  Here
// a CTA of 128 threads owns a tz x ty tile of (z, y) columns and marches `chunk`
// x-planes.  Per plane it
//   A. evaluates the link data of its sites and of the low y and z halo once,
//      into shared memory (x-backward data stay in registers): 6 sincos and 6
//      sines, on the integer pipe (dtrig.cuh);
//   B. updates its sites, on the FP64 pipe (2 instructions per SM and cycle),
//      which bounds the step: about 310 FP64 instructions a site where the
//      one-pass kernel has 560.
// Three CTAs share an SM (168 registers): while one is in A, another is in B.
// Planes are staged in shared memory two ahead by cp.async, so a site's
// neighbours are read from HBM once.  (An Abelian-Higgs form of this kernel was
// 10-25 % slower than the two-pass step: there the FP64 pipe is busy 90 % of the
// update already, and the march adds the halo's FP64 work.)
//
// The tile is chosen per lattice so that few lanes idle (march_tile): with 32x4
// tiles a 101-wide row would leave 21 % of the FP64 pipe's lanes empty.
//
// STRICT: every expression is the one-pass kernel's, evaluated on the same
// operands: same doubles.  Otherwise (LAT_F64_FAST, compiled with multiply-add
// contraction) sin(P_yx) = -sin(P_xy) and likewise zx, zy.
#pragma once

#include <cuda_pipeline.h>

#include "ah_twopass.cuh"
#include "tiled_step.cuh"

namespace lat {

constexpr int M64_THREADS = 128;
constexpr int M64_STAGES = 3;
constexpr int M64_NC = 7;       // components
constexpr int M64_NL = 12;      // link-data arrays
constexpr int M64_SITES = 256;  // staged positions of a plane (two per thread)

struct MarchTile {
    int tz, ty;      // tile extents, tz*ty <= 128, (tz+2)*(ty+2) <= M64_SITES
    int ntz, nty;    // tiles along z and y
};

// The tile with the least work for an hy x hz region: threads launched plus the
// halo's link evaluations (about a third of a site's cost each).
inline MarchTile march_tile(int hy, int hz)
{
    MarchTile best{};
    double cost = 1e300;
    for (int n = (hz + 63) / 64; n <= (hz + 7) / 8 || n == (hz + 63) / 64; ++n) {
        const int tz = (hz + n - 1) / n;
        int ty = M64_THREADS / tz;
        while (ty > 1 && (tz + 2) * (ty + 2) > M64_SITES) --ty;
        if (ty > hy) ty = hy;
        const int ntz = (hz + tz - 1) / tz, nty = (hy + ty - 1) / ty;
        ty = (hy + nty - 1) / nty;   // even rows
        const double t = (double)ntz * nty * (32 * ((tz * ty + 31) / 32) + 0.33 * (tz + ty));
        if (t < cost) {
            cost = t;
            best = MarchTile{tz, ty, ntz, nty};
        }
    }
    return best;
}

// x-planes per CTA: the least work for the SM with the most CTAs, where a CTA
// costs its planes and about 0.8 more (it starts with the link data of the
// plane before its first) and an SM needs three CTAs at a time to keep the FP64
// pipe busy (96^3: 16 planes; 24, two CTAs per SM, cost 10 % more).
inline int march64_chunk(const MarchTile& m, int hx)
{
    const int64_t tiles = (int64_t)m.ntz * m.nty;
    int best = 1;
    double cost = 1e300;
    for (int c : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64}) {
        const int64_t per_sm = (tiles * ((hx + c - 1) / c) + 151) / 152;
        const double t = (c + 0.8) * (per_sm < 3 ? 3 : per_sm);
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

inline int64_t march64_ctas(const Geom& g)
{
    const MarchTile m = march_tile(g.hiy - g.loy, g.hiz - g.loz);
    const int c = march64_chunk(m, g.hix - g.lox);
    return (int64_t)m.ntz * m.nty * ((g.hix - g.lox + c - 1) / c);
}

// doubles of shared memory: staged planes, link data, the diagnostics' sums
inline size_t march64_smem(const MarchTile& m)
{
    const size_t stage = (size_t)(m.tz + 2) * (m.ty + 2) * M64_NC * M64_STAGES;
    const size_t links = (size_t)(m.tz + 1) * (m.ty + 1) * M64_NL;
    return sizeof(double) * (stage + links + 8);
}

// link data in shared memory: per scalar cos/sin of q*theta_y and q*theta_z,
// then the sines of P_xy, P_xz, P_yz and (strict) P_zy
enum { M64_PXY = 8, M64_PXZ, M64_PYZ, M64_PZY };
constexpr __device__ int m64_cy(int f) { return 4 * f; }
constexpr __device__ int m64_sy(int f) { return 4 * f + 1; }
constexpr __device__ int m64_cz(int f) { return 4 * f + 2; }
constexpr __device__ int m64_sz(int f) { return 4 * f + 3; }

// The Moore update of one site in moore_step.cuh's order of operations.
struct MooreSite {
    double v[2][2], vp[2][2][3], vm[2][2][3], qv[2][2];
    double th[3], thm[3], qth[3];
    double cs[2][3], sn[2][3], csm[2][3], snm[2][3];
    // sines of the plaquettes at the site and at their backward neighbours
    double sPxy, sPxz, sPyz, sPyx, sPzx, sPzy, sPxy_m, sPxz_m, sPyz_m, sPyx_m, sPzx_m, sPzy_m;
    double cPxy, cPxz, cPyz, divPast;
};

template <bool DIAG, bool RECIP>
__device__ __forceinline__ void moore_site(const MooreSite& m, const StepCoef& c, const DiagOut& d, double (&next)[7],
                                           double& divNow, double& e_site, double& g_site)
{
    const double q[2] = {c.q1, c.q2};
    double mag[2];
#pragma unroll
    for (int fi = 0; fi < 2; ++fi) mag[fi] = m.v[fi][0] * m.v[fi][0] + m.v[fi][1] * m.v[fi][1];
    const double pot[2] = {c.halfLambda * (mag[0] - c.etaSq) + c.halfLambda12 * (mag[1] - c.eta2Sq),
                           c.halfLambda2 * (mag[1] - c.eta2Sq) + c.halfLambda12 * (mag[0] - c.etaSq)};
    double acc[2][2];
#pragma unroll
    for (int fi = 0; fi < 2; ++fi) {
#pragma unroll
        for (int comp = 0; comp < 2; ++comp) {
            double num[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (comp == 0)
                    num[a] = minus_twice(m.cs[fi][a] * m.vp[fi][0][a] + m.sn[fi][a] * m.vp[fi][1][a], m.v[fi][0])
                           + m.csm[fi][a] * m.vm[fi][0][a] - m.snm[fi][a] * m.vm[fi][1][a];
                else
                    num[a] = minus_twice(m.cs[fi][a] * m.vp[fi][1][a] - m.sn[fi][a] * m.vp[fi][0][a], m.v[fi][1])
                           + m.csm[fi][a] * m.vm[fi][1][a] + m.snm[fi][a] * m.vm[fi][0][a];
            }
            double tt = lap_minus<RECIP>(num[0], num[1], num[2], pot[fi] * m.v[fi][comp], c);
            if (nonzero(c.fric)) tt = tt - c.fric * cdiv(m.v[fi][comp] - m.qv[fi][comp], c.dt, c.inv_dt);
            acc[fi][comp] = tt;
        }
    }
    double cur[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double cf[2];
#pragma unroll
        for (int fi = 0; fi < 2; ++fi) {
            const double val = m.cs[fi][a] * (m.v[fi][1] * m.vp[fi][0][a] - m.v[fi][0] * m.vp[fi][1][a])
                             + m.sn[fi][a] * (m.v[fi][0] * m.vp[fi][0][a] + m.v[fi][1] * m.vp[fi][1][a]);
            cf[fi] = d.charge_current ? q[fi] * val : val;
        }
        cur[a] = cf[0] + cf[1];
    }
    double tt[3] = {sub_sdiv<RECIP>(c.m2gg * cur[0], m.sPxy - m.sPxy_m, c.dy2, c.inv_dy2),
                    sub_sdiv<RECIP>(c.m2gg * cur[1], m.sPyx - m.sPyx_m, c.dx2, c.inv_dx2),
                    sub_sdiv<RECIP>(c.m2gg * cur[2], m.sPzx - m.sPzx_m, c.dx2, c.inv_dx2)};
    tt[0] = sub_sdiv<RECIP>(tt[0], m.sPxz - m.sPxz_m, c.dz2, c.inv_dz2);
    tt[1] = sub_sdiv<RECIP>(tt[1], m.sPyz - m.sPyz_m, c.dz2, c.inv_dz2);
    tt[2] = sub_sdiv<RECIP>(tt[2], m.sPzy - m.sPzy_m, c.dy2, c.inv_dy2);
    if (nonzero(c.damp)) {
#pragma unroll
        for (int a = 0; a < 3; ++a) tt[a] = tt[a] - c.damp * cdiv(m.th[a] - m.qth[a], c.dt, c.inv_dt);
    }
    divNow = 0;
    if (DIAG || d.store_div)
        divNow = sdiv<RECIP>(m.th[0] - m.thm[0], c.dx2, c.inv_dx2) + sdiv<RECIP>(m.th[1] - m.thm[1], c.dy2, c.inv_dy2)
               + sdiv<RECIP>(m.th[2] - m.thm[2], c.dz2, c.inv_dz2);
    if constexpr (DIAG) {
        const double dd[3] = {c.dx, c.dy, c.dz}, idd[3] = {c.inv_dx, c.inv_dy, c.inv_dz};
        double pt[2][2], pd[2][3][2];
#pragma unroll
        for (int fi = 0; fi < 2; ++fi) {
            pt[fi][0] = cdiv(m.v[fi][0] - m.qv[fi][0], c.dt, c.inv_dt);
            pt[fi][1] = cdiv(m.v[fi][1] - m.qv[fi][1], c.dt, c.inv_dt);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                pd[fi][a][0] = sdiv<RECIP>(m.v[fi][0] - m.csm[fi][a] * m.vm[fi][0][a] + m.snm[fi][a] * m.vm[fi][1][a], dd[a], idd[a]);
                pd[fi][a][1] = sdiv<RECIP>(m.v[fi][1] - m.csm[fi][a] * m.vm[fi][1][a] - m.snm[fi][a] * m.vm[fi][0][a], dd[a], idd[a]);
            }
        }
        double tdc = 0, fc = 0, gauss = 0;
        const double t0 = m.th[0] - m.qth[0], t1 = m.th[1] - m.qth[1], t2 = m.th[2] - m.qth[2];
        if (d.energy_form == LAT_ENERGY_MPI) {
            const double a0 = cdiv(t0, c.dt, c.inv_dt), a1 = cdiv(t1, c.dt, c.inv_dt), a2 = cdiv(t2, c.dt, c.inv_dt);
            tdc = 0.5 * (a0 * a0 + a1 * a1 + a2 * a2);
            fc = cdiv(1 - m.cPxy, c.gxy2, c.inv_gxy2) + cdiv(1 - m.cPxz, c.gxz2, c.inv_gxz2)
               + cdiv(1 - m.cPyz, c.gyz2, c.inv_gyz2);
        }
        if (nonzero(c.g)) {
            const double divThetat = cdiv(divNow - m.divPast, c.dt, c.inv_dt);
            gauss = cdiv(divThetat, c.g, c.inv_g)
                  - c.twog * (q[0] * (m.v[0][1] * pt[0][0] - m.v[0][0] * pt[0][1])
                              + q[1] * (m.v[1][1] * pt[1][0] - m.v[1][0] * pt[1][1]));
            if (d.energy_form != LAT_ENERGY_MPI) {
                const double a0 = cdiv(t0, c.gdtdx, c.inv_gdtdx), a1 = cdiv(t1, c.gdtdy, c.inv_gdtdy),
                             a2 = cdiv(t2, c.gdtdz, c.inv_gdtdz);
                tdc = 0.5 * (a0 * a0 + a1 * a1 + a2 * a2);
                const double Fxy = cdiv(1 - m.cPxy, c.gxy2, c.inv_gxy2);
                const double Fxz = cdiv(1 - m.cPxz, c.gxz2, c.inv_gxz2);
                const double Fyz = cdiv(1 - m.cPyz, c.gyz2, c.inv_gyz2);
                fc = Fxy + Fxz + Fyz;
            }
        }
        const double m1 = mag[0] - c.etaSq, m2 = mag[1] - c.eta2Sq;
        const double ed = pt[0][0] * pt[0][0] + pt[0][1] * pt[0][1] + pd[0][0][0] * pd[0][0][0] + pd[0][0][1] * pd[0][0][1]
                        + pd[0][1][0] * pd[0][1][0] + pd[0][1][1] * pd[0][1][1] + pd[0][2][0] * pd[0][2][0]
                        + pd[0][2][1] * pd[0][2][1] + pt[1][0] * pt[1][0] + pt[1][1] * pt[1][1]
                        + pd[1][0][0] * pd[1][0][0] + pd[1][0][1] * pd[1][0][1] + pd[1][1][0] * pd[1][1][0]
                        + pd[1][1][1] * pd[1][1][1] + pd[1][2][0] * pd[1][2][0] + pd[1][2][1] * pd[1][2][1] + tdc + fc
                        + c.quarterLambda * (m1 * m1) + c.quarterLambda2 * (m2 * m2) + c.halfLambda12e * m1 * m2;
        if (d.energy_form == LAT_ENERGY_MPI) e_site = ed * c.dx * c.dy * c.dz;
        else e_site = c.dV * ed;
        g_site = __longlong_as_double(__double_as_longlong(gauss) & 0x7fffffffffffffffll);
    }
#pragma unroll
    for (int fi = 0; fi < 2; ++fi)
#pragma unroll
        for (int comp = 0; comp < 2; ++comp)
            next[2 * fi + comp] = twice_minus(m.v[fi][comp], m.qv[fi][comp]) + c.dt2 * acc[fi][comp];
#pragma unroll
    for (int a = 0; a < 3; ++a) next[4 + a] = twice_minus(m.th[a], m.qth[a]) + c.dt2 * tt[a];
}

// DIAG: the CTA's energy and |G| sums go to d.partials[2*blockIdx.x].
template <bool STRICT, bool DIAG, bool RECIP>
__global__ void __launch_bounds__(M64_THREADS, 3)
moore_march_kernel(const Geom g, const MarchTile mt, const Fields<double, 7> f, const StepCoef c, const DiagOut d,
                   const int chunk)
{
    chain_wait();
    constexpr int NC = M64_NC, TH = 4;
    extern __shared__ __align__(16) double sm64[];
    const int P = mt.tz + 2, SP = P * (mt.ty + 2);   // staged row pitch, plane
    const int Q = mt.tz + 1, LP = Q * (mt.ty + 1);   // link row pitch, plane
    double* const L = sm64 + (size_t)M64_STAGES * NC * SP;
    const int tid = threadIdx.x;
    const int tiles = mt.ntz * mt.nty;
    const int bz = (int)blockIdx.x / tiles, bt = (int)blockIdx.x - bz * tiles;
    const int k0 = g.loz + (bt % mt.ntz) * mt.tz, j0 = g.loy + (bt / mt.ntz) * mt.ty;
    const int ib = g.lox + bz * chunk, ie = min(ib + chunk, g.hix);
    const int wz = min(mt.tz, g.hiz - k0), wy = min(mt.ty, g.hiy - j0);
    const int ly = tid / mt.tz, lz = tid - ly * mt.tz;
    const bool active = ly < wy && lz < wz;
    const int jj = active ? j0 + ly : j0, kk = active ? k0 + lz : k0;
    const int o = active ? (ly + 1) * P + lz + 1 : P + 1;       // own staged position
    const int lo = active ? (ly + 1) * Q + lz + 1 : Q + 1;      // own link position
    const double q[2] = {c.q1, c.q2};

    // staged positions of this thread: in-plane source offset, or -1
    int src[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int s = tid + r * M64_THREADS, hy = s / P, hz = s - hy * P;
        src[r] = (s < SP && hy <= wy + 1 && hz <= wz + 1)
                     ? wrap_idx(j0 - 1 + hy, g.ny) * g.nz + wrap_idx(k0 - 1 + hz, g.nz) : -1;
    }
    auto stage = [&](int b, int pi) {
        const int base = pi * g.syz;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (src[r] >= 0) {
                double* dst = sm64 + (size_t)b * NC * SP + tid + r * M64_THREADS;
#pragma unroll
                for (int m = 0; m < NC; ++m) __pipeline_memcpy_async(dst + m * SP, f.now[m] + (base + src[r]), 8);
            }
        __pipeline_commit();
    };
    stage(0, wrap_idx(ib, g.nx));
    stage(1, wrap_idx(ib + 1, g.nx));

    // plane ib-1 of the own column: what plane ib reads as x-backward data
    double cxm[2], sxm[2], vm[4], bxy, bxz, txm;   // bxy, bxz: sin P_yx, P_zx there (FAST: of P_xy, P_xz)
    {
        const int im = wrap_idx(ib - 1, g.nx), i0 = wrap_idx(ib, g.nx);
        const int s = (im * g.ny + jj) * g.nz + kk, sxp = (i0 * g.ny + jj) * g.nz + kk;
        const int syp = (im * g.ny + wrap_idx(jj + 1, g.ny)) * g.nz + kk;
        const int szp = (im * g.ny + jj) * g.nz + wrap_idx(kk + 1, g.nz);
        const double tx = f.now[TH][s], ty = f.now[TH + 1][s], tz = f.now[TH + 2][s];
        const double tyxp = f.now[TH + 1][sxp], tzxp = f.now[TH + 2][sxp], txyp = f.now[TH][syp], txzp = f.now[TH][szp];
#pragma unroll
        for (int a = 0; a < 2; ++a) dsincos(q[a] * tx, &sxm[a], &cxm[a]);
        if constexpr (STRICT) {
            bxy = dsin(ty + txyp - tyxp - tx);
            bxz = dsin(tz + txzp - tzxp - tx);
        } else {
            bxy = dsin(tx + tyxp - txyp - ty);
            bxz = dsin(tx + tzxp - txzp - tz);
        }
        txm = tx;
#pragma unroll
        for (int m = 0; m < 4; ++m) vm[m] = f.now[m][s];
    }
    double e_acc = 0, g_acc = 0;
    int cur = 0;
    for (int i = ib; i < ie; ++i) {
        const int nxt = cur == 2 ? 0 : cur + 1, nn = nxt == 2 ? 0 : nxt + 1;
        __pipeline_wait_prior(0);   // planes i and i+1 have landed
        __syncthreads();            // for everybody; plane i-1 and its link data are done with
        if (i + 1 < ie) stage(nn, wrap_idx(i + 2, g.nx));
        const double* const S = sm64 + (size_t)cur * NC * SP;
        const double* const X = sm64 + (size_t)nxt * NC * SP;
        const int s = (i * g.ny + jj) * g.nz + kk;
        double past[NC];
#pragma unroll
        for (int m = 0; m < NC; ++m) past[m] = active ? f.past[m][s] : 0.0;

        // ---- A: link data
        const double tx = S[TH * SP + o], ty = S[(TH + 1) * SP + o], tz = S[(TH + 2) * SP + o];
        double cx[2], sx[2], sPxy, sPxz, sPyx = 0, sPzx = 0, cP[3] = {0, 0, 0};
        {
            const double tyxp = X[(TH + 1) * SP + o], tzxp = X[(TH + 2) * SP + o];
            const double txyp = S[TH * SP + o + P], tzyp = S[(TH + 2) * SP + o + P];
            const double txzp = S[TH * SP + o + 1], tyzp = S[(TH + 1) * SP + o + 1];
            double cv, sv, sPyz;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                dsincos(q[a] * tx, &sx[a], &cx[a]);
                dsincos(q[a] * ty, &sv, &cv);
                if (active) L[m64_cy(a) * LP + lo] = cv, L[m64_sy(a) * LP + lo] = sv;
                dsincos(q[a] * tz, &sv, &cv);
                if (active) L[m64_cz(a) * LP + lo] = cv, L[m64_sz(a) * LP + lo] = sv;
            }
            const double Pxy = tx + tyxp - txyp - ty, Pxz = tx + tzxp - txzp - tz, Pyz = ty + tzyp - tyzp - tz;
            if constexpr (DIAG) {
                dsincos(Pxy, &sPxy, &cP[0]);
                dsincos(Pxz, &sPxz, &cP[1]);
                dsincos(Pyz, &sPyz, &cP[2]);
            } else {
                sPxy = dsin(Pxy);
                sPxz = dsin(Pxz);
                sPyz = dsin(Pyz);
            }
            if (active) L[M64_PXY * LP + lo] = sPxy, L[M64_PXZ * LP + lo] = sPxz, L[M64_PYZ * LP + lo] = sPyz;
            if constexpr (STRICT) {
                sPyx = dsin(ty + txyp - tyxp - tx);
                sPzx = dsin(tz + txzp - tzxp - tx);
                const double sPzy = dsin(tz + tyzp - tzyp - ty);
                if (active) L[M64_PZY * LP + lo] = sPzy;
            }
        }
        // low halo: the row y = j0-1, then the column z = k0-1, one position a
        // thread, taken from the last threads (the first ones' warps are full)
        for (int h = M64_THREADS - 1 - tid; h < wz + wy; h += M64_THREADS) {
            const bool row = h < wz;
            const int hy = row ? 0 : h - wz + 1, hz = row ? h + 1 : 0;     // staged position
            const int p = hy * P + hz, l = hy * Q + hz;
            const double ax = S[TH * SP + p], ay = S[(TH + 1) * SP + p], az = S[(TH + 2) * SP + p];
            const double azyp = S[(TH + 2) * SP + p + P], ayzp = S[(TH + 1) * SP + p + 1];
            const double b = row ? ay : az;
            double cv, sv;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                dsincos(q[a] * b, &sv, &cv);
                L[(row ? m64_cy(a) : m64_cz(a)) * LP + l] = cv;
                L[(row ? m64_sy(a) : m64_sz(a)) * LP + l] = sv;
            }
            // row: P_xy; column: P_xz
            const double fx = row ? X[(TH + 1) * SP + p] : X[(TH + 2) * SP + p];
            const double gx = row ? S[TH * SP + p + P] : S[TH * SP + p + 1];
            L[(row ? M64_PXY : M64_PXZ) * LP + l] = dsin(ax + fx - gx - b);
            // row: P_zy (FAST: P_yz); column: P_yz
            if constexpr (STRICT)
                L[(row ? M64_PZY : M64_PYZ) * LP + l] = row ? dsin(az + ayzp - azyp - ay) : dsin(ay + azyp - ayzp - az);
            else
                L[M64_PYZ * LP + l] = dsin(ay + azyp - ayzp - az);
        }
        __syncthreads();

        // ---- B: update
        double e_site = 0, g_site = 0;
        if (active) {
            double next[NC], divNow;
            MooreSite v;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const double* const F = S + (2 * a + k) * SP + o;
                    v.v[a][k] = F[0];
                    v.vp[a][k][0] = X[(2 * a + k) * SP + o], v.vm[a][k][0] = vm[2 * a + k];
                    v.vp[a][k][1] = F[P], v.vm[a][k][1] = F[-P];
                    v.vp[a][k][2] = F[1], v.vm[a][k][2] = F[-1];
                    v.qv[a][k] = past[2 * a + k];
                }
                v.cs[a][0] = cx[a], v.sn[a][0] = sx[a], v.csm[a][0] = cxm[a], v.snm[a][0] = sxm[a];
                v.cs[a][1] = L[m64_cy(a) * LP + lo], v.sn[a][1] = L[m64_sy(a) * LP + lo];
                v.csm[a][1] = L[m64_cy(a) * LP + lo - Q], v.snm[a][1] = L[m64_sy(a) * LP + lo - Q];
                v.cs[a][2] = L[m64_cz(a) * LP + lo], v.sn[a][2] = L[m64_sz(a) * LP + lo];
                v.csm[a][2] = L[m64_cz(a) * LP + lo - 1], v.snm[a][2] = L[m64_sz(a) * LP + lo - 1];
            }
            v.th[0] = tx, v.th[1] = ty, v.th[2] = tz;
            v.thm[0] = txm, v.thm[1] = S[(TH + 1) * SP + o - P], v.thm[2] = S[(TH + 2) * SP + o - 1];
            v.qth[0] = past[4], v.qth[1] = past[5], v.qth[2] = past[6];
            v.sPxy = sPxy, v.sPxz = sPxz, v.sPyz = L[M64_PYZ * LP + lo];
            v.sPxy_m = L[M64_PXY * LP + lo - Q], v.sPxz_m = L[M64_PXZ * LP + lo - 1], v.sPyz_m = L[M64_PYZ * LP + lo - 1];
            if constexpr (STRICT) {
                v.sPyx = sPyx, v.sPzx = sPzx, v.sPzy = L[M64_PZY * LP + lo];
                v.sPyx_m = bxy, v.sPzx_m = bxz, v.sPzy_m = L[M64_PZY * LP + lo - Q];
            } else {
                v.sPyx = -v.sPxy, v.sPzx = -v.sPxz, v.sPzy = -v.sPyz;
                v.sPyx_m = -bxy, v.sPzx_m = -bxz, v.sPzy_m = -L[M64_PYZ * LP + lo - Q];
            }
            if constexpr (DIAG) {
                v.cPxy = cP[0], v.cPxz = cP[1], v.cPyz = cP[2];
                if (nonzero(c.g)) v.divPast = reinterpret_cast<const double*>(d.divbuf)[s];
            }
            moore_site<DIAG, RECIP>(v, c, d, next, divNow, e_site, g_site);
            if (d.store_div) reinterpret_cast<double*>(d.divbuf)[s] = divNow;
            if (d.write) {
#pragma unroll
                for (int m = 0; m < NC; ++m) f.past[m][s] = next[m];
            }
        }
        if constexpr (DIAG) {
            e_acc += e_site;
            g_acc += g_site;
        }
        // x-backward data of the next plane
#pragma unroll
        for (int a = 0; a < 2; ++a) cxm[a] = cx[a], sxm[a] = sx[a];
#pragma unroll
        for (int m = 0; m < 4; ++m) vm[m] = S[m * SP + o];
        bxy = STRICT ? sPyx : sPxy;
        bxz = STRICT ? sPzx : sPxz;
        txm = tx;
        cur = nxt;
    }
    __pipeline_wait_prior(0);
    if constexpr (DIAG) {
        double* const red = L + (size_t)LP * M64_NL;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            e_acc += __shfl_down_sync(0xffffffffu, e_acc, w);
            g_acc += __shfl_down_sync(0xffffffffu, g_acc, w);
        }
        if ((tid & 31) == 0) {
            red[tid >> 5] = e_acc;
            red[4 + (tid >> 5)] = g_acc;
        }
        __syncthreads();
        if (tid == 0) {
            d.partials[2 * blockIdx.x] = red[0] + red[1] + red[2] + red[3];
            d.partials[2 * blockIdx.x + 1] = red[4] + red[5] + red[6] + red[7];
        }
    }
}

template <bool STRICT>
cudaError_t launch_moore_march_t(const Geom& g, const Fields<double, 7>& f, const StepCoef& c, const DiagOut& d,
                                 bool diag, bool recip, cudaStream_t st)
{
    const MarchTile m = march_tile(g.hiy - g.loy, g.hiz - g.loz);
    const int chunk = march64_chunk(m, g.hix - g.lox);
    const size_t smem = march64_smem(m);
    const unsigned grid = (unsigned)march64_ctas(g);
    cudaError_t e = cudaSuccess;
    auto go = [&](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        e = launch_chained(kernel, grid, M64_THREADS, smem, st, g, m, f, c, d, chunk);
    };
    if (diag) {
        if (recip) go(moore_march_kernel<STRICT, true, true>);
        else go(moore_march_kernel<STRICT, true, false>);
    } else {
        if (recip) go(moore_march_kernel<STRICT, false, true>);
        else go(moore_march_kernel<STRICT, false, false>);
    }
    return e;
}

}  // namespace lat
