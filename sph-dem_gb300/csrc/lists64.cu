/*
 * FP64 passes of the fluid particles, over the neighbour lists:
 *   k_force64   calcForce (calcViscForce, calcPressForce, calcNormal,
 *               calcBoundaryForces) with calcOmega and the Courant / viscous /
 *               accel dt conditions      sphIncompress.h:899-972, sph.h:438-451, 545-918
 *   k_dddt64    calcDddtDudt with calcOmega           sphIncompress.h:783-851
 *   k_invm      calcInvM + inverseSym (CORRECTED_GRADIENT)
 *                                                     sph.h:393-434, vect.h:49-111
 *   k_reinit_h, k_reinit_dens
 *               the density re-initialisation of start(): ten rounds of
 *               calcHFromDens + calcDensity           sphIncompress.cpp:19-35,
 *                                                     sph.h:1823-1825, 1172-1184
 *
 * The lists are those of the mixed path (k_nlist): built in FP32 with a proven
 * error bound, candidates in doubt decided by the reference's FP64 predicate,
 * so they hold the reference's neighbours exactly.  A particle with more
 * neighbours than the lists are deep, and a handle without lists, takes its
 * bucket stencil instead, testing every candidate in FP64.
 *
 * These passes are bound by the FP64 pipe (2 lanes per SM and cycle): what
 * counts is FP64 instructions per pair.  Hence no candidate is tested here
 * (the stencil holds six times the neighbours), the Wendland gradient has its
 * closed form F(r, h) = -10 C / h^(d+2) (2 - r/h)^3 (no division by q), square
 * roots and reciprocals start from an FP32 estimate, constant factors are
 * applied to the sums, calcOmega shares the loop, and G lanes share a particle
 * so that every SM has its part of the pairs.  Before (a thread scanning its
 * stencil) / now, us: coupled step of 69,758 particles, force 24,856 / 1,136,
 * continuity and Omega 16,795 / 502 (3D, ~85 neighbours); dam break of 23,018
 * (2D), force 742 / 90, continuity 385 / 31; of 8,753 with CORRECTED_GRADIENT
 * and density re-initialisation, k_invm twice 1,577 / 101, k_reinit_dens 1,192 / 79.
 */
#include "fp64.cuh"
#include "mixed.cuh"

namespace sphdem {
namespace {

/* lanes per particle: about five pairs each in 2D, eleven in 3D (1D has few).
 * Force / continuity, us, with 2 / 4 / 8 lanes in 2D: 1,418 particles 38 / 27 / 21
 * and 20 / 14 / 12, 23,018 80 / 90 / 104 and 35 / 31 / 37; with 4 / 8 / 16 in 3D:
 * 69,758 1142 / 1142 / 1295 and 493 / 509 / 529.  One number per dimension: in 2D 8
 * lanes would take 8 us off a step of 1,418 particles and add 20 to one of 23,018. */
template <int ND>
constexpr int LANES64 = ND == 3 ? 8 : (ND == 2 ? 4 : 1);

struct Lists64 {
    const int *nbr, *ncnt;
    int64_t ld;
};

/* every neighbour b of particle a (position ra, smoothing length ha; hrow: the
 * smoothing lengths of the neighbour predicate): body(b, dx, r2) with dx = r_a -
 * image(r_b); a lane visits every G-th list entry, or (no list) lane 0 the
 * bucket stencil */
template <int ND, int G, class Body>
__device__ __forceinline__ void visit_neighbours(const DevCfg &c, const DevState &s, const DevGlobals *g, const Lists64 &L,
                                                 const int *__restrict__ start, const int *__restrict__ skey, int a,
                                                 const double *ra, double ha, const double *hrow, int sub, Body &&body) {
    const int cnt = L.nbr ? L.ncnt[a] : -1;
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    if (cnt >= 0) {
        int cc[3] = {0, 0, 0};
        decode<ND>(skey[a], dims, cc);
        bool seam = false; /* the bucket has a neighbour across a periodic face */
#pragma unroll
        for (int d = 0; d < ND; d++) seam |= c.periodic[d] && (cc[d] == 0 || cc[d] == dims[d] - 1);
        for (int j = sub; j < cnt; j += G) {
            const int e = L.nbr[nl_at(a, j, L.ld)], b = e & B_MASK;
            double rb[ND], dx[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int d = 0; d < ND; d++) rb[d] = s.row(FD_R + d)[b];
            if (seam) {
                int o[3];
                nl_decode_code(e >> B_BITS, o);
#pragma unroll
                for (int d = 0; d < ND; d++) {
                    const int t = cc[d] + o[d];
                    rb[d] = image_pos(rb[d], t < 0 ? -1 : (t >= dims[d] ? 1 : 0), c.rmin[d], c.rmax[d]);
                }
            }
#pragma unroll
            for (int d = 0; d < ND; d++) dx[d] = dsub(ra[d], rb[d]);
            double r2 = dx[0] * dx[0];
#pragma unroll
            for (int d = 1; d < ND; d++) r2 = fma(dx[d], dx[d], r2);
            body(b, dx, r2);
        }
    } else if (sub == 0) {
        const CellCoord cc = decode_cell(skey[a], dims, ND);
        scan_cells(cc, dims, c.periodic, ND, start, 0, [&](int b, const int *sh) {
            const bool shifted = sh[0] | sh[1] | sh[2];
            if (b == a && !shifted) return;
            double dx[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int d = 0; d < ND; d++) dx[d] = dsub(ra[d], image_pos(s.row(FD_R + d)[b], sh[d], c.rmin[d], c.rmax[d]));
            const double r2 = exact_len2(dx, ND), hb = hrow[b], t = 2.0 * (ha > hb ? ha : hb);
            if (r2 > dmul(t, t) || (shifted && !image_exists(s.irow(FI_GCODE)[b], sh, ND))) return;
            body(b, dx, r2);
        });
    }
}

/* calcNormal, sph.h:736-779 */
__device__ void calc_normal(const DevCfg &c, const DevState &s, int b, const double *dx, double r,
                                            double *normp, double *normt) {
    double n1[3] = {0, 0, 0}, n2[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) {
        n1[d] = s.row(FD_N1 + d)[b];
        n2[d] = s.row(FD_N2 + d)[b];
        normt[d] = c.nd == 3 ? s.row(FD_N3 + d)[b] : 0.0;
    }
    const bool n2zero = n2[0] == 0 && n2[1] == 0 && n2[2] == 0;
    if (n2zero) {
        for (int d = 0; d < 3; d++) normp[d] = n1[d];
        return;
    }
    const float rdot1 = dot3(dx, n1, c.nd);
    const float rdot2 = dot3(dx, n2, c.nd);
    const float rntest = r * r * dot3(n1, n2, c.nd) - rdot1 * rdot2;
    if (rntest <= 0) {
        for (int d = 0; d < c.nd; d++) normp[d] = dx[d] / r;
        return;
    }
    const int con = s.irow(FI_CONCAVE)[b] ? 1 : -1;
    if (con * (rdot1 - rdot2) > 0)
        for (int d = 0; d < 3; d++) normp[d] = n1[d];
    else
        for (int d = 0; d < 3; d++) normp[d] = n2[d];
}

/* calcNormal + calcBoundaryForces, sph.h:736-918: the force of repulsive
 * boundary particle b (at dx, relative velocity dv) added to fb */
__device__ __noinline__ void boundary64(const DevCfg *__restrict__ cp, const DevState &s, int b, double ma, double dx0,
                                        double dx1, double dx2, double r, double dv0, double dv1, double dv2, double *fb) {
    const DevCfg &c = *cp;
    const double dx[3] = {dx0, dx1, dx2}, dv[3] = {dv0, dv1, dv2}, mb = s.row(FD_MASS)[b];
    double normp[3] = {0, 0, 0}, normt[3] = {0, 0, 0};
    calc_normal(c, s, b, dx, r, normp, normt);
    const double rperp = dot3(normp, dx, c.nd);
    double rt[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) rt[d] = dx[d] - rperp * normp[d];
    double pt0, pt1;
    const double rDelP = 1.0 / (c.bfac * c.psep);
    if (c.nd == 3) {
        pt0 = fabs(dot3(rt, normt, 3));
        const double cr[3] = {rt[1] * normt[2] - rt[2] * normt[1], rt[2] * normt[0] - rt[0] * normt[2],
                              rt[0] * normt[1] - rt[1] * normt[0]};
        pt1 = sqrt(dot3(cr, cr, 3));
    } else {
        pt0 = sqrt(dot3(rt, rt, c.nd));
        pt1 = 0;
    }
    const double pd0 = pt0 * rDelP, pd1 = pt1 * rDelP;
    if (!(pd0 <= 1.0 && pd1 <= 1.0)) return;
    const double q = fabs(rperp) / (1.0 * c.psep);
    if (!(q < 2.0)) return;
    const double pesky = 0.25 * (1 + cos(c.pi * pd0)) * (1 + cos(c.pi * pd1));
    const int beta = dot3(dx, dv, c.nd) < 0 ? 1 : 0;
    const double bigA = 0.01 * (c.spsound * c.spsound) - beta * c.spsound * dot3(dv, normp, c.nd);
    const double bfact = 1.0 / fabs(rperp);
    const double QIN = 2.0 / 3.0;
    double bforce = 0.0;
    if (q <= QIN) bforce = bfact * QIN;
    else if (q <= 1.0) bforce = bfact * (2.0 * q - 1.5 * q * q);
    else bforce = bfact * 0.5 * ((2.0 - q) * (2.0 - q));
    const double bigR = bigA * bforce;
    const double amassrat = 2.0 * ma / (ma + mb);
    const int sign = rperp < 0 ? -1 : 1;
    for (int d = 0; d < c.nd; d++) fb[d] += sign * amassrat * normp[d] * bigR * pesky * 1.0;
}

/* gradW with CORRECTED_GRADIENT (sph.h:325-326): invM ((dr F - sumGrad/sum)/sum),
 * with M = invM / sum and cs = sumGrad / sum */
template <int ND>
struct Cg64 {
    double m[ND * ND], cs[ND];
    __device__ __forceinline__ void load(const double *cg, int64_t cap, int64_t a) {
        const double sum = cg[CG_S * cap + a];
#pragma unroll
        for (int k = 0; k < ND * ND; k++) m[k] = cg[(CG_M + k) * cap + a] / sum;
#pragma unroll
        for (int d = 0; d < ND; d++) cs[d] = cg[(CG_C + d) * cap + a];
    }
    __device__ __forceinline__ void apply(const double *dx, double F, double *out) const {
        double t[ND];
#pragma unroll
        for (int d = 0; d < ND; d++) t[d] = fma(dx[d], F, -cs[d]);
#pragma unroll
        for (int i = 0; i < ND; i++) {
            double v = m[i * ND] * t[0];
#pragma unroll
            for (int j = 1; j < ND; j++) v = fma(m[i * ND + j], t[j], v);
            out[i] = v;
        }
    }
};

/* d/dh of the kernel (calcOmega, sph.h:438-451): C (10 q^2 - d t (1 + 2q)) t^3 /
 * h^(d+1), t = 2 - q cut at 0, without C / h^(d+1) */
template <int ND>
__device__ __forceinline__ double omega_poly(double q, double t3) {
    return fma(fma(10.0 + 2.0 * ND, q, -3.0 * ND), q, -2.0 * ND) * t3;
}
/* Omega from the sum of omega_poly over the neighbours, a's own term -2 d C m 2^3 / h^(d+1) */
template <int ND>
__device__ __forceinline__ double omega_of(const DevCfg &c, double sum, double ma, double ha, double ihn, double ih, double dens) {
    return 1.0 + ha * (ihn * ih * c.wcon) * (sum - 16.0 * ND * ma) / (dens * ND);
}

template <int ND, bool CG>
__global__ void __launch_bounds__(BLK) k_force64(DevCfg c, const DevCfg *__restrict__ cp, DevState s, Lists64 L,
                                                 const int *__restrict__ start, const int *__restrict__ skey, DevGlobals *g,
                                                 const double *__restrict__ cg, int64_t n) {
    constexpr int G = LANES64<ND>;
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const int ta = a < n ? s.irow(FI_IAM)[a] : -1;
    const bool act = is_sph_or_sphb(ta);
    double ndt = DBL_MAX;
    double ha = 1.0, iha = 1.0, densa = 1.0;
    double fp[ND], fv[ND], fb[3] = {0, 0, 0}, om = 0.0, fq = 0.0;
#pragma unroll
    for (int d = 0; d < ND; d++) fp[d] = fv[d] = 0.0;
    const bool var_h = c.var_h(), anti = !(c.flags & SPHDEM_F_NO_ANTICLUMPING);
    /* F = kf / h^(d+2) t^3; without CORRECTED_GRADIENT kf is applied to the sums */
    const double kf = -10.0 * c.wcon, kp = CG ? kf : 1.0;
    if (act) {
        double ra[3] = {0, 0, 0}, va[ND];
#pragma unroll
        for (int d = 0; d < ND; d++) {
            ra[d] = s.row(FD_R + d)[a];
            va[d] = s.row(FD_VHAT + d)[a];
        }
        ha = s.row(FD_H)[a];
        iha = s.row(FD_IH)[a];
        densa = s.row(FD_DENS)[a];
        const double cFa = kp * s.row(FD_IHN2)[a], pdr2a = s.row(FD_PDR2)[a], ma = s.row(FD_MASS)[a];
        Cg64<ND> cw;
        if (CG) cw.load(cg, s.cap, a);
        const double k_anti_inv = anti ? 1.0 / c.k_anti : 0.0;
        double hmin = DBL_MAX;                 /* smallest hav of the fluid pairs */
        double hbest = DBL_MAX, vbest = 1.0;   /* the pair with the smallest hav / vsig */
        const double twoc0 = 2.0 * c.spsound;
        visit_neighbours<ND, G>(c, s, g, L, start, skey, (int)a, ra, ha, s.row(FD_H), sub, [&](int b, const double *dx, double r2) {
            const int tb = s.irow(FI_IAM)[b];
            double ri;
            const double r = sqrt_pos(r2, &ri);
            const double hb = s.row(FD_H)[b];
            double t = positive_part(fma(-r, iha, 2.0));
            const double ta3 = t * t * t;
            t = positive_part(fma(-r, s.row(FD_IH)[b], 2.0));
            const double Fb = (kp * s.row(FD_IHN2)[b]) * (t * t * t);
            const double Fa = cFa * ta3;
            const double F = var_h ? Fa + Fb : 0.5 * (Fa + Fb);   /* var_h: twice the mean */
            const double mb = s.row(FD_MASS)[b], densb = s.row(FD_DENS)[b];
            const bool fluid_b = is_sph_or_sphb(tb);
            if (var_h && fluid_b) om = fma(mb, omega_poly<ND>(r * iha, ta3), om);
            /* gradients of a's and b's kernel, and their mean */
            double gA[ND], gB[ND];
            if (CG) {
                cw.apply(dx, Fa, gA);
                cw.apply(dx, Fb, gB);
                if (!var_h)
#pragma unroll
                    for (int d = 0; d < ND; d++) gA[d] = gB[d] = 0.5 * (gA[d] + gB[d]);
            }
            if (fluid_b) {
                /* calcPressForce, sph.h:692-734 */
                const double pdr2b = s.row(FD_PDR2)[b];
                if (CG) {
#pragma unroll
                    for (int d = 0; d < ND; d++) fp[d] -= mb * (pdr2a * gA[d] + pdr2b * gB[d]);
                } else {
                    const double w = -mb * (var_h ? fma(pdr2a, Fa, pdr2b * Fb) : (pdr2a + pdr2b) * F);
#pragma unroll
                    for (int d = 0; d < ND; d++) fp[d] = fma(w, dx[d], fp[d]);
                }
                if (anti) {
                    const double kdw = wK(r / (0.5 * (ha + hb)), c.wcon) * k_anti_inv, k2 = kdw * kdw;
                    fq -= mb * (0.01 * fabs(pdr2a + pdr2b) * (k2 * k2));
                }
            }
            if (ta == T_SPH && tb != T_DEM && tb != T_DEMB) {
                /* calcViscForce, sph.h:579-666 */
                double dv[ND];
#pragma unroll
                for (int d = 0; d < ND; d++) dv[d] = va[d] - s.row(FD_VHAT + d)[b];
                const double hav = 0.5 * (ha + hb);
                /* the mean gradient is dx cM, or gM */
                double cM = var_h ? 0.5 * F : F, gM[ND];
                if (CG)
#pragma unroll
                    for (int d = 0; d < ND; d++) gM[d] = 0.5 * (gA[d] + gB[d]);
                if (c.visc == SPHDEM_VISC_MORRIS) {
                    double dg = r2 * cM;
                    if (CG) {
                        dg = dx[0] * gM[0];
#pragma unroll
                        for (int d = 1; d < ND; d++) dg = fma(dx[d], gM[d], dg);
                    }
                    const double num = c.liq_dem() ? 2.0 * c.viscosity * c.dens : c.viscosity * (densa + densb);
                    const double sc = (mb * num) * dg * rcp_pos((densa * densb) * fma(0.01 * hav, hav, r2));
#pragma unroll
                    for (int d = 0; d < ND; d++) fv[d] = fma(dv[d], sc, fv[d]);
                } else if (c.visc == SPHDEM_VISC_MONAGHAN || c.visc == SPHDEM_VISC_ARTIFICIAL) {
                    double vdr = dx[0] * dv[0];
#pragma unroll
                    for (int d = 1; d < ND; d++) vdr = fma(dx[d], dv[d], vdr);
                    const bool mon = c.visc == SPHDEM_VISC_MONAGHAN;
                    /* artificial viscosity acts on approaching pairs only */
                    const double viss = mon || vdr < 0 ? vdr * ri : 0.0;
                    const double vsig = mon ? (c.liq_dem() ? 0.0 : twoc0 + 2.0 * fabs(viss))
                                            : (vdr < 0 ? twoc0 - 4.0 * viss : 0.0);
                    const double sv = mb * viss * vsig * (mon ? c.alpha_mon : c.alpha_art) * rcp_pos(densa + densb);
#pragma unroll
                    for (int d = 0; d < ND; d++) fv[d] = CG ? fma(sv, gM[d], fv[d]) : fma(sv * cM, dx[d], fv[d]);
                    /* hav / vsig < hbest / vbest (vsig = 0 bounds nothing) */
                    if (hav * vbest < hbest * vsig) {
                        hbest = hav;
                        vbest = vsig;
                    }
                }
                hmin = min_pos(hmin, hav);
            }
            if (is_boundary(tb)) {
                double dv[3] = {0, 0, 0};
#pragma unroll
                for (int d = 0; d < ND; d++) dv[d] = va[d] - s.row(FD_VHAT + d)[b];
                boundary64(cp, s, b, ma, dx[0], dx[1], dx[2], r, dv[0], dv[1], dv[2], fb);
            }
        });
        if (hmin < DBL_MAX) {
            if (c.visc == SPHDEM_VISC_MORRIS) ndt = 0.6 * hmin / twoc0;
            else if (hbest < DBL_MAX) ndt = 0.6 * hbest / vbest;
            const double vdc = c.visc == SPHDEM_VISC_MONAGHAN ? 0.06 : 0.125;
            ndt = fmin(ndt, vdc * (hmin * hmin) / c.viscosity);
        }
    }
    const bool walls = __any_sync(0xffffffffu, fb[0] != 0.0 || fb[1] != 0.0 || fb[2] != 0.0);
#pragma unroll
    for (int d = 0; d < ND; d++) {
        fp[d] = lane_sum<G>(fp[d]);
        fv[d] = lane_sum<G>(fv[d]);
        if (walls) fb[d] = lane_sum<G>(fb[d]);
    }
    if (var_h) om = lane_sum<G>(om);
    if (anti) fq = lane_sum<G>(fq);
    if (act && sub == 0) {
        double sc = CG ? 1.0 : kf;
        if (var_h) {
            /* every gradient of a's sums carries 1 / Omega_a */
            const double omega = omega_of<ND>(c, om, s.row(FD_MASS)[a], ha, s.row(FD_IHN)[a], iha, densa);
            s.row(FD_OMEGA)[a] = omega;
            sc /= omega;
        }
        double f2 = 0.0;
#pragma unroll
        for (int d = 0; d < ND; d++) {
            const double fpd = fma(fp[d], sc, fq), fvd = fv[d] * sc;
            s.row(FD_FP + d)[a] += fpd;
            if (c.visc != SPHDEM_VISC_ARTIFICIAL) s.row(FD_FV + d)[a] += fvd;
            s.row(FD_FB + d)[a] += fb[d];
            const double f = s.row(FD_F + d)[a] + ((fpd + fvd) + fb[d]);
            s.row(FD_F + d)[a] = f;
            f2 = fma(f, f, f2);
        }
        /* accelCondition, sph.h:566-568 */
        ndt = fmin(ndt, 0.25 * sqrt(ha / sqrt(f2)));
    }
    block_min_atomic(ndt, &g->new_dt_bits);
}

template <int ND, bool CG>
__global__ void __launch_bounds__(BLK) k_dddt64(DevCfg c, DevState s, Lists64 L, const int *__restrict__ start,
                                                const int *__restrict__ skey, const DevGlobals *g,
                                                const double *__restrict__ cg, int64_t n) {
    constexpr int G = LANES64<ND>;
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const bool act = a < n && is_sph_or_sphb(s.irow(FI_IAM)[a]);
    const bool var_h = c.var_h();
    const double kf = -10.0 * c.wcon, kp = CG ? kf : 1.0;
    double acc = 0.0, om = 0.0, ha = 1.0, iha = 1.0;
    if (act) {
        double ra[3] = {0, 0, 0}, va[ND];
#pragma unroll
        for (int d = 0; d < ND; d++) {
            ra[d] = s.row(FD_R + d)[a];
            va[d] = s.row(FD_VHAT + d)[a];
        }
        ha = s.row(FD_H)[a];
        iha = s.row(FD_IH)[a];
        const double cFa = kp * s.row(FD_IHN2)[a];
        Cg64<ND> cw;
        if (CG) cw.load(cg, s.cap, a);
        visit_neighbours<ND, G>(c, s, g, L, start, skey, (int)a, ra, ha, s.row(FD_H), sub, [&](int b, const double *dx, double r2) {
            const int tb = s.irow(FI_IAM)[b];
            if (is_boundary(tb) || tb == T_DEM) return;
            const double r = sqrt_pos(r2), mb = s.row(FD_MASS)[b];
            double t = positive_part(fma(-r, iha, 2.0));
            const double ta3 = t * t * t, Fa = cFa * ta3;
            double Fb = 0.0;
            if (var_h) {
                if (is_sph_or_sphb(tb)) om = fma(mb, omega_poly<ND>(r * iha, ta3), om);
            } else {
                t = positive_part(fma(-r, s.row(FD_IH)[b], 2.0));
                Fb = (kp * s.row(FD_IHN2)[b]) * (t * t * t);
            }
            double dv[ND], vdr = 0.0;
#pragma unroll
            for (int d = 0; d < ND; d++) dv[d] = va[d] - s.row(FD_VHAT + d)[b];
            if (CG) {
                double wa[ND], wb[ND];
                cw.apply(dx, Fa, wa);
                if (!var_h) cw.apply(dx, Fb, wb);
#pragma unroll
                for (int d = 0; d < ND; d++) vdr = fma(dv[d], var_h ? wa[d] : 0.5 * (wa[d] + wb[d]), vdr);
                acc = fma(mb, vdr, acc);
            } else {
                vdr = dv[0] * dx[0];
#pragma unroll
                for (int d = 1; d < ND; d++) vdr = fma(dv[d], dx[d], vdr);
                acc = fma(mb * vdr, Fa + Fb, acc); /* constant h: twice the mean */
            }
        });
    }
    acc = lane_sum<G>(acc);
    if (var_h) om = lane_sum<G>(om);
    if (!act || sub) return;
    double sc = CG ? 1.0 : (var_h ? kf : 0.5 * kf);
    if (var_h) {
        const double omega =
            omega_of<ND>(c, om, s.row(FD_MASS)[a], ha, s.row(FD_IHN)[a], iha, s.row(FD_DENS)[a]);
        s.row(FD_OMEGA)[a] = omega;
        sc /= omega;
    }
    s.row(FD_DDDT)[a] += acc * sc;
}

/* inverseSym (vect.h:49-111): adjugate over determinant; identity when the
 * determinant is 0.  1D (which the reference does not define) inverts the
 * scalar. */
__device__ void inverse_sym(double *a, int nd) {
    if (nd == 1) {
        a[0] = a[0] != 0.0 ? 1.0 / a[0] : 1.0;
        return;
    }
    if (nd == 2) {
        const double A = a[0], B = a[1], C = a[2], D = a[3];
        const double det = dsub(dmul(A, D), dmul(B, C));
        if (det != 0.0) {
            a[0] = D / det;
            a[1] = -B / det;
            a[2] = -C / det;
            a[3] = A / det;
        } else {
            a[0] = 1.0;
            a[1] = 0.0;
            a[2] = 0.0;
            a[3] = 1.0;
        }
        return;
    }
    const double A0 = a[0], B0 = a[1], C0 = a[2], D0 = a[3], E0 = a[4], F0 = a[5], G0 = a[6], H0 = a[7], K0 = a[8];
    const double cA = dsub(dmul(E0, K0), dmul(F0, H0)), cB = dsub(dmul(F0, G0), dmul(D0, K0));
    const double cC = dsub(dmul(D0, H0), dmul(E0, G0)), cD = dsub(dmul(C0, H0), dmul(B0, K0));
    const double cE = dsub(dmul(A0, K0), dmul(C0, G0)), cF = dsub(dmul(B0, G0), dmul(A0, H0));
    const double cG = dsub(dmul(B0, F0), dmul(C0, E0)), cH = dsub(dmul(C0, D0), dmul(A0, F0));
    const double cK = dsub(dmul(A0, E0), dmul(B0, D0));
    const double Z = dadd(dadd(dmul(A0, cA), dmul(B0, dsub(dmul(F0, G0), dmul(K0, D0)))), dmul(C0, cC));
    if (Z != 0.0) {
        const double o[9] = {cA, cD, cG, cB, cE, cH, cC, cF, cK};
        for (int k = 0; k < 9; k++) a[k] = o[k] / Z;
    } else {
        for (int k = 0; k < 9; k++) a[k] = (k % 4 == 0) ? 1.0 : 0.0;
    }
}

/* calcInvM (sph.h:393-434) of every sph / sphBoundary particle over the
 * neighbours of the last rebuild: sum = (m/rho) W(0,h) + sum dvol W(r/hav,hav),
 * sumGrad = sum dvol dr F(r/hav,hav), M = -sum dvol (dr F - sumGrad/sum)/sum (x) dr,
 * invM = M^-1 (identity without neighbours).  One pass: with S = sumGrad/sum,
 * M = -(sum dvol F dr (x) dr - S (x) sum dvol dr) / sum. */
template <int ND>
__global__ void __launch_bounds__(BLK) k_invm(DevCfg c, DevState s, Lists64 L, const int *__restrict__ start,
                                              const int *__restrict__ skey, const DevGlobals *g, double *cg, int64_t n) {
    constexpr int G = LANES64<ND>;
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const bool act = a < n && is_sph_or_sphb(s.irow(FI_IAM)[a]);
    double sum = 0.0, sg[ND], sd[ND], mm[ND * (ND + 1) / 2];
    int nn = 0;
#pragma unroll
    for (int d = 0; d < ND; d++) sg[d] = sd[d] = 0.0;
#pragma unroll
    for (int k = 0; k < ND * (ND + 1) / 2; k++) mm[k] = 0.0;
    const double kf = -10.0 * c.wcon;
    if (act) {
        double ra[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < ND; d++) ra[d] = s.row(FD_R + d)[a];
        const double ha = s.row(FD_H)[a];
        visit_neighbours<ND, G>(c, s, g, L, start, skey, (int)a, ra, ha, s.row(FD_H), sub, [&](int b, const double *dx, double r2) {
            nn++;
            if (!is_sph_or_sphb(s.irow(FI_IAM)[b])) return;
            const double dvol = s.row(FD_MASS)[b] * rcp_pos(s.row(FD_DENS)[b]);
            /* F(q, hav) and W(q, hav) of the pair (sph.h:74-80, 306-308) */
            const double ih = rcp_pos(0.5 * (ha + s.row(FD_H)[b])), q = sqrt_pos(r2) * ih;
            const double t = positive_part(2.0 - q), t3 = t * t * t;
            double ihn = ih;
#pragma unroll
            for (int d = 1; d < ND; d++) ihn *= ih;
            sum = fma(dvol * ihn, c.wcon * (t3 * t) * fma(2.0, q, 1.0), sum);
            /* at r = 0 the gradient of the pair is zero as dr is */
            const double vF = dvol * (kf * (ihn * ih * ih)) * t3;
            int k = 0;
#pragma unroll
            for (int i = 0; i < ND; i++) {
                const double w = vF * dx[i];
                sg[i] += w;
                sd[i] = fma(dvol, dx[i], sd[i]);
#pragma unroll
                for (int j = i; j < ND; j++, k++) mm[k] = fma(w, dx[j], mm[k]);
            }
        });
    }
    sum = lane_sum<G>(sum);
#pragma unroll
    for (int d = 0; d < ND; d++) {
        sg[d] = lane_sum<G>(sg[d]);
        sd[d] = lane_sum<G>(sd[d]);
    }
#pragma unroll
    for (int k = 0; k < ND * (ND + 1) / 2; k++) mm[k] = lane_sum<G>(mm[k]);
#pragma unroll
    for (int o = 1; o < G; o <<= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    if (!act || sub) return;
    sum += (s.row(FD_MASS)[a] / s.row(FD_DENS)[a]) * (s.row(FD_IHN)[a] * wK(0.0, c.wcon));
    double m[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (nn == 0) {
        for (int i = 0; i < ND; i++) m[i * ND + i] = 1.0;
    } else {
        int k = 0;
        for (int i = 0; i < ND; i++)
            for (int j = i; j < ND; j++, k++) {
                m[i * ND + j] = -(mm[k] - (sg[i] / sum) * sd[j]) / sum;
                if (j != i) m[j * ND + i] = -(mm[k] - (sg[j] / sum) * sd[i]) / sum;
            }
        inverse_sym(m, ND);
    }
    const int64_t cap = s.cap;
    for (int k = 0; k < ND * ND; k++) cg[(CG_M + k) * cap + a] = m[k];
    for (int d = 0; d < ND; d++) cg[(CG_C + d) * cap + a] = sg[d] / sum;
    cg[CG_S * cap + a] = sum;
}

/* Density re-initialisation (sphIncompress.cpp:19-35).  The neighbour lists
 * of the reference are built lazily after the first calcHFromDens, so the
 * neighbour predicate uses that first h (kept in hp) through all ten
 * rounds, while calcDensity uses each round's own h.  The lists hold the pairs
 * within 2 max(hp) as long as no hp outgrew the buckets; `wide` is set when
 * one did, and every particle then scans its buckets. */
__global__ void k_reinit_h(DevCfg c, DevState s, DevGlobals *g, double *hp, int *wide, int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(s.irow(FI_IAM)[a])) return;
    const double m = s.row(FD_MASS)[a], rho = s.row(FD_DENS)[a];
    const double x = c.precision == SPHDEM_PREC_MIXED ? m * recip(c, rho) : m / rho;
    const double h = smoothing_length(c, x);
    s.row(FD_H)[a] = h;
    hp[a] = h;
    if (!(h <= g->sr)) *wide = 1;
}

/* R_KEEP distances and masses of a lane's neighbours stay in registers from
 * round to round; a lane with more reads the others again */
constexpr int R_KEEP = 8;
template <int ND>
__global__ void __launch_bounds__(BLK) k_reinit_dens(DevCfg c, DevState s, Lists64 L, const int *__restrict__ start,
                                                     const int *__restrict__ skey, const DevGlobals *g, const double *hp,
                                                     const int *wide, int64_t n) {
    constexpr int G = LANES64<ND>;
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const bool act = a < n && is_sph_or_sphb(s.irow(FI_IAM)[a]);
    if (*wide) L.nbr = nullptr;
    double ra[3] = {0, 0, 0}, ma = 1.0, h = 1.0, rho = 1.0, hpa = 1.0;
    double rk[R_KEEP], mk[R_KEEP];
    int kept = 0, seen = 0;
#pragma unroll
    for (int k = 0; k < R_KEEP; k++) rk[k] = mk[k] = 0.0;
    auto visit = [&](auto &&body) {
        visit_neighbours<ND, G>(c, s, g, L, start, skey, (int)a, ra, hpa, hp, sub, [&](int b, const double *, double r2) {
            if (!is_sph_or_sphb(s.irow(FI_IAM)[b])) return;
            body(b, r2);
        });
    };
    if (act) {
#pragma unroll
        for (int d = 0; d < ND; d++) ra[d] = s.row(FD_R + d)[a];
        ma = s.row(FD_MASS)[a];
        hpa = hp[a];
        h = s.row(FD_H)[a];
        rho = s.row(FD_DENS)[a];
        visit([&](int b, double r2) {
            const double r = sqrt_pos(r2), mb = s.row(FD_MASS)[b];
#pragma unroll
            for (int k = 0; k < R_KEEP; k++)
                if (k == seen) {
                    rk[k] = r;
                    mk[k] = mb;
                }
            seen++;
        });
        kept = min(seen, R_KEEP);
    }
    for (int round = 0; round < 10; round++) {
        if (round > 0) {
            const double x = c.precision == SPHDEM_PREC_MIXED ? ma * recip(c, rho) : ma / rho;
            h = smoothing_length(c, x);
        }
        const double ih = recip(c, h);
        double sum = 0.0; /* of m (2 - q)^4 (1 + 2q) */
#pragma unroll
        for (int k = 0; k < R_KEEP; k++)
            if (k < kept) {
                const double q = rk[k] * ih, t = positive_part(2.0 - q), t2 = t * t;
                sum = fma(mk[k] * (t2 * t2), fma(2.0, q, 1.0), sum);
            }
        if (seen > R_KEEP) {
            int i = 0;
            visit([&](int b, double r2) {
                if (i++ < R_KEEP) return;
                const double q = sqrt_pos(r2) * ih, t = positive_part(2.0 - q), t2 = t * t;
                sum = fma(s.row(FD_MASS)[b] * (t2 * t2), fma(2.0, q, 1.0), sum);
            });
        }
        sum = lane_sum<G>(sum);
        double ihn = ih;
#pragma unroll
        for (int d = 1; d < ND; d++) ihn *= ih;
        rho = (ihn * c.wcon) * fma(16.0, ma, sum);
    }
    if (act && sub == 0) {
        s.row(FD_H)[a] = h;
        h_derived(c, s, a);
        s.row(FD_DENS)[a] = rho;
    }
}

/* the records of the FP32 searches: offset in the particle's own bucket and h,
 * type and ghost code, a DEM particle's place in the SPH grid; in the middle
 * phase the Shepard sums start at zero */
template <int ND>
__global__ void k_pack_pos(DevCfg c, DevState s, const int *__restrict__ skey, const DevGlobals *__restrict__ g,
                           float4 *__restrict__ P0, int *__restrict__ tg, float4 *__restrict__ DS, int middle, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = s.irow(FI_IAM)[i];
    tg[i] = (t & 0xff) | (s.irow(FI_GCODE)[i] << 8);
    if (t == T_DEAD) return;
    const bool dem = c.liq_dem() && t == T_DEM;
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    int cc[3] = {0, 0, 0};
    if (dem) decode<ND>(skey[i] - g->n_sph_cells, c.ddims, cc);
    else decode<ND>(skey[i], dims, cc);
    float off[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < ND; d++)
        off[d] = (float)(s.row(FD_R + d)[i] - (dem ? dem_origin(c, d, cc[d]) : sph_origin(c, g, d, cc[d])));
    if (dem && middle) s.row(FD_SHEP)[i] = 0.0;
    if (dem && !middle && DS) DS[i] = dem_in_sph_grid<ND>(c, s, g, i);
    P0[i] = make_float4(off[0], off[1], off[2], (float)s.row(FD_H)[i]);
}

Lists64 lists_of(const sphdem_ctx *c) {
    const int depth = c->cfg.precision == SPHDEM_PREC_MIXED ? c->mx_maxn : c->f64_maxn;
    return depth > 0 ? Lists64{c->mx_nbr, c->mx_ncnt, depth} : Lists64{nullptr, nullptr, 0};
}

template <int ND>
int blocks64(int64_t n) {
    return grid_for(n * LANES64<ND>, BLK);
}

}  // namespace

void pack_positions(sphdem_ctx *c, bool middle) {
#define L_(ND)                                                                                                   \
    SPHDEM_LAUNCH(c, "pack_pos", k_pack_pos<ND>, grid_for(c->n, 256), 256, 0, c->cfg, c->A, c->buf.skey, c->g, \
                  c->mx_pos, c->mx_tg, c->mx_ds, (int)middle, c->n)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
}

void run_lists64(sphdem_ctx *c, bool middle) {
    if (c->f64_maxn > 0 || c->f64_dem) pack_positions(c, middle);
    if (c->f64_maxn > 0) mixed::nlist(c, c->f64_maxn, true);
}

void run_force(sphdem_ctx *c) {
    const double *cg = corrected_gradient(c) ? c->cg : nullptr;
#define LK_(ND, CGF)                                                                                              \
    SPHDEM_LAUNCH(c, "force_fp64", (k_force64<ND, CGF>), blocks64<ND>(c->n), BLK, 0, c->cfg, c->dcfg, c->A,     \
                  lists_of(c), c->buf.start, c->buf.skey, c->g, cg, c->n)
#define L_(ND)              \
    do {                    \
        if (cg)             \
            LK_(ND, true);  \
        else                \
            LK_(ND, false); \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LK_
}

void run_dddt(sphdem_ctx *c) {
    const double *cg = corrected_gradient(c) ? c->cg : nullptr;
#define LK_(ND, CGF)                                                                                              \
    SPHDEM_LAUNCH(c, "dddt_fp64", (k_dddt64<ND, CGF>), blocks64<ND>(c->n), BLK, 0, c->cfg, c->A, lists_of(c),   \
                  c->buf.start, c->buf.skey, c->g, cg, c->n)
#define L_(ND)              \
    do {                    \
        if (cg)             \
            LK_(ND, true);  \
        else                \
            LK_(ND, false); \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LK_
}

void run_invm(sphdem_ctx *c) {
#define L_(ND)                                                                                                    \
    SPHDEM_LAUNCH(c, "invm_fp64", k_invm<ND>, blocks64<ND>(c->n), BLK, 0, c->cfg, c->A, lists_of(c), c->buf.start, \
                  c->buf.skey, c->g, c->cg, c->n)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
}

void run_reinit_density(sphdem_ctx *c) {
    rebuild(c);
    const Lists64 L = lists_of(c);
    SPHDEM_CUDA_CHECK(cudaMemsetAsync(c->reinit_wide, 0, sizeof(int), c->stream));
    SPHDEM_LAUNCH(c, "reinit_h", k_reinit_h, grid_for(c->n, 256), 256, 0, c->cfg, c->A, c->g, c->hpred, c->reinit_wide,
                  c->n);
    if (L.nbr) {
        pack_positions(c, false);
        mixed::nlist(c, (int)L.ld, true);
    }
#define L_(ND)                                                                                                    \
    SPHDEM_LAUNCH(c, "reinit_dens_fp64", k_reinit_dens<ND>, blocks64<ND>(c->n), BLK, 0, c->cfg, c->A, L,         \
                  c->buf.start, c->buf.skey, c->g, c->hpred, c->reinit_wide, c->n)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
}

}  // namespace sphdem
