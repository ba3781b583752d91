/*
 * FP64 EOS and DEM time step, and the coupling and contact passes of an FP64
 * handle whose lengths lie outside FP32's range, so that it has no FP32 records
 * to search (coupling.cu): one thread per target particle over the buckets,
 * every candidate tested in FP64.
 *
 *   k_porosity  calcPorosity + calcShepSum        sph.h:1323-1341, 1303-1320
 *   k_dem_drag  calcDEMtoSPHDrag + finalisePorosity + setPorosityForBoundary
 *                                                 sph.h:1343-1362, 1289-1296, 1263-1265
 *   k_eos       calcPressSpsoundPdr2               sphIncompress.h:863-896
 *   k_dem_end   calcFPI + calcParticleDrag + calcDEMContacts
 *                                                 sph.h:1708-1792, 1575-1631, 1676-1706
 * The fluid's own passes (force, continuity, calcOmega, calcInvM, density
 * re-initialisation) are in lists64.cu.
 *
 * Neighbour sets are those of the reference exactly: the same 3^d bucket
 * stencil, the FP64 predicate |r_a-r_b|^2 <= (2 max(h_a,h_b))^2 evaluated
 * without FMA in blitz's order, periodic images only where the reference
 * holds a ghost copy, and the asymmetric SPH->DEM bucket rule of
 * dataLL.cpp:1154-1190.  Within a bucket, neighbours are visited in tag
 * order, which is the reference's own order for non-periodic cases.
 *
 * The Shepard sum is the only scatter of the reference (SPH particles add
 * into their DEM neighbours); it stays a scatter here with FP64 atomics.
 *
 * Roofline: FP64-pipe-bound (this GPU's FP64 rate is a small fraction of
 * its FP32 rate); this path is the plain-FP64 baseline.
 */
#include <cfloat>

#include "fp64.cuh"

namespace sphdem {
namespace {

constexpr int BLK = 128;

/* ---------------------------------------------------------------------- */
/* SPH -> DEM coupling search (calcNeighboursCoupling for non-DEM particles) */
template <class Body>
__device__ __forceinline__ void scan_coupling(const DevCfg &c, const DevState &s, const int *start,
                                              int dem_base, const double *ra, Body &&body) {
    int cs[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) cs[d] = ref_dem_cell(ra[d], c, d);
    const CellCoord cc = dem_cell_of(c, ra);
    scan_cells(cc, c.ddims, c.periodic, c.nd, start, dem_base, [&](int b, const int *sh) {
        if (s.irow(FI_IAM)[b] != T_DEM) return;
        int cd[3] = {0, 0, 0};
        double rb[3] = {0, 0, 0};
        const bool shifted = (sh[0] | sh[1] | sh[2]) != 0;
        for (int d = 0; d < c.nd; d++) {
            rb[d] = image_pos(s.row(FD_R + d)[b], sh[d], c.rmin[d], c.rmax[d]);
            cd[d] = shifted ? ref_dem_cell(rb[d], c, d) : s.irow(FI_RDC0 + d)[b];
        }
        if (!coupling_rule(cs, cd, c)) return;
        double dx[3] = {0, 0, 0};
        for (int d = 0; d < c.nd; d++) dx[d] = dsub(ra[d], rb[d]);
        const double r2 = exact_len2(dx, c.nd);
        if (!(r2 < c.rc2)) return;  /* beyond Rc every contribution is exactly 0 */
        if (shifted && !image_exists(s.irow(FI_GCODE)[b], sh, c.nd)) return;
        body(b, dx, r2);
    });
}

__global__ void k_porosity(DevCfg c, DevState s, const int *start, const DevGlobals *g, int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(s.irow(FI_IAM)[a])) return;
    const int dem_base = g->n_sph_cells;
    double ra[3] = {0, 0, 0}, va[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) {
        ra[d] = s.row(FD_R + d)[a];
        va[d] = s.row(FD_VHAT + d)[a];
    }
    const double dvol = s.row(FD_MASS)[a] / s.row(FD_DENS)[a];
    double por = 0.0, dpordt = 0.0, gp[3] = {0, 0, 0};
    scan_coupling(c, s, start, dem_base, ra, [&](int b, const double *dx, double r2) {
        const double r = sqrt(r2);
        const double q = r * c.two_over_rc;
        const double Wa = c.c_ihn * wK(q, c.wcon);
        por += c.por_incr * Wa;
        if (r != 0.0) {
            double dv[3] = {0, 0, 0};
            for (int d = 0; d < c.nd; d++) dv[d] = va[d] - s.row(FD_VHAT + d)[b];
            const double Fq = c.c_ihn2 * wdK(q, c.wcon) / q;
            dpordt -= c.dem_vol * dot3(dv, dx, c.nd) * Fq;
            for (int d = 0; d < c.nd; d++) gp[d] += c.dem_vol * dx[d] * Fq;
        }
        atomicAdd(&s.row(FD_SHEP)[b], dvol * Wa);
    });
    s.row(FD_POR)[a] = por;
    s.row(FD_DPORDT)[a] = dpordt;
    for (int d = 0; d < 3; d++) s.row(FD_GPOR + d)[a] = gp[d];
}

__global__ void k_zero_dem_shep(DevState s, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.irow(FI_IAM)[i] == T_DEM) s.row(FD_SHEP)[i] = 0.0;
}

__global__ void k_dem_drag(DevCfg c, DevState s, const int *start, const DevGlobals *g, int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    const int t = s.irow(FI_IAM)[a];
    if (is_boundary(t)) {
        s.row(FD_POR)[a] = 1.0;
        return;
    }
    if (!is_sph_or_sphb(t)) return;
    const int dem_base = g->n_sph_cells;
    double ra[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) ra[d] = s.row(FD_R + d)[a];
    const double densa = s.row(FD_DENS)[a];
    const double rdens = c.nd == 2 ? (1.0 / (2.0 * c.dem_radius)) / densa : 1.0 / densa;
    double fd[3] = {0, 0, 0};
    scan_coupling(c, s, start, dem_base, ra, [&](int b, const double *dx, double r2) {
        const double r = sqrt(r2);
        const double w = c.c_ihn * wK(r * c.two_over_rc, c.wcon);
        const double mb = s.row(FD_MASS)[b], sb = s.row(FD_SHEP)[b];
        for (int d = 0; d < c.nd; d++) fd[d] -= mb * rdens * s.row(FD_FDRAG + d)[b] * w / sb;
    });
    for (int d = 0; d < c.nd; d++) {
        s.row(FD_FDRAG + d)[a] = fd[d];
        s.row(FD_F + d)[a] += fd[d];
    }
    double por = 1.0 - s.row(FD_POR)[a];
    if (por < 0.37) {
        por = 0.37;
        s.row(FD_DPORDT)[a] = 0.0;
        for (int d = 0; d < 3; d++) s.row(FD_GPOR + d)[a] = 0.0;
    }
    s.row(FD_POR)[a] = por;
}

/* ---------------------------------------------------------------------- */
__global__ void k_eos(DevCfg c, DevState s, int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(s.irow(FI_IAM)[a])) return;
    const double densa = s.row(FD_DENS)[a];
    double press;
    double x = c.liq_dem() ? densa / (c.refd * s.row(FD_POR)[a]) : densa / c.refd;
    if (!c.liq_dem() || c.gamma == 7.0) {
        const double x2 = x * x;
        press = c.prb * (x2 * x2 * x2 * x - 1.0);
    } else {
        press = c.prb * (pow(x, c.gamma) - 1.0);
    }
    s.row(FD_PRESS)[a] = press;
    s.row(FD_PDR2)[a] = press / (densa * densa);
}

__global__ void k_dem_accel(DevCfg c, DevState s, DevGlobals *g, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double ndt = DBL_MAX;
    if (i < n && s.irow(FI_IAM)[i] == T_DEM) {
        double f[3] = {0, 0, 0};
        for (int d = 0; d < c.nd; d++) f[d] = s.row(FD_F + d)[i];
        ndt = 0.25 * sqrt(s.row(FD_H)[i] / sqrt(dot3(f, f, c.nd)));
    }
    block_min_atomic(ndt, &g->new_dt_bits);
}

/* ---------------------------------------------------------------------- */
__device__ __forceinline__ double radius_of(const DevCfg &c, const DevState &s, int i) {
    const double r = s.row(FD_RADIUS)[i];
    return r > 0.0 ? r : c.dem_radius;
}

__global__ void k_dem_end(DevCfg c, DevState s, const int *start, const DevGlobals *g, int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (s.irow(FI_IAM)[a] != T_DEM) return;
    const GridInfo gi = load_grid(g);
    double ra[3] = {0, 0, 0}, va[3] = {0, 0, 0}, f[3] = {0, 0, 0}, fpv[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) {
        ra[d] = s.row(FD_R + d)[a];
        va[d] = s.row(FD_VHAT + d)[a];
        f[d] = s.row(FD_F + d)[a];
        fpv[d] = s.row(FD_FP + d)[a];
    }
    const double ha = s.row(FD_H)[a], ma = s.row(FD_MASS)[a];
    /* calcFPI over the SPH buckets (calcNeighboursCoupling for a DEM particle) */
    double sum = 0, fdens = 0, por = 0;
    double ff[3] = {0, 0, 0}, fpfb[3] = {0, 0, 0}, fv[3] = {0, 0, 0}, fdr[3] = {0, 0, 0}, fvel[3] = {0, 0, 0};
    const CellCoord cs = sph_cell_of(c, gi, ra);
    scan_cells(cs, gi.sdims, c.periodic, c.nd, start, 0, [&](int b, const int *sh) {
        double dx[3], r2;
        if (!pair_geom(c, s, b, sh, ra, ha, dx, r2)) return;
        if (s.irow(FI_IAM)[b] == T_BOUNDARY) return;
        const double r = sqrt(r2);
        const double mb = s.row(FD_MASS)[b];
        const double dvol = mb / s.row(FD_DENS)[b];
        const double q = r * s.row(FD_IH)[b];
        const double Wab = s.row(FD_IHN)[b] * wK(q, c.wcon);
        const double dvWab = dvol * Wab;
        for (int d = 0; d < c.nd; d++) {
            fpfb[d] += mb * Wab * (s.row(FD_FP + d)[b] + s.row(FD_FB + d)[b]);
            fv[d] += mb * Wab * s.row(FD_FV + d)[b];
            fv[d] += dvWab * s.row(FD_FV + d)[b];
            ff[d] += dvWab * s.row(FD_F + d)[b];
            fdr[d] += dvWab * s.row(FD_FDRAG + d)[b];
            fvel[d] += dvWab * s.row(FD_VHAT + d)[b];
        }
        por += dvWab * s.row(FD_POR)[b];
        fdens += Wab * mb;
        sum += dvWab;
    });
    double fdrag_out[3] = {0, 0, 0};
    if (sum > 0.5) {
        const double rsum = 1.0 / sum;
        for (int d = 0; d < c.nd; d++) {
            ff[d] *= rsum;
            fpfb[d] *= rsum;
            fv[d] *= rsum;
            fdr[d] *= rsum;
            fvel[d] *= rsum;
        }
        fdens *= rsum;
        por *= rsum;
        for (int d = 0; d < c.nd; d++) {
            s.row(FD_FB + d)[a] = fpfb[d];
            s.row(FD_FV + d)[a] = fv[d];
        }
        /* calcParticleDrag, Di Felice (sph.h:1575-1631) */
        double dv[3] = {0, 0, 0};
        for (int d = 0; d < c.nd; d++) dv[d] = por * (fvel[d] - va[d]);
        const double vdiff = sqrt(dot3(dv, dv, c.nd));
        double fd[3] = {0, 0, 0};
        if (vdiff != 0) {
            const double A = c.pi * (c.dem_radius * c.dem_radius);
            const double Re = (2.0 * c.dem_radius / c.viscosity) * vdiff;
            const double lg = 1.5 - log10(Re);
            const double dragGamma = 3.7 - 0.65 * exp(-(lg * lg) / 2.0);
            const double cc0 = 0.63 + 4.8 / sqrt(Re);
            const double C = cc0 * cc0;
            const double sc = (1.0 / 2.0) * A * C * vdiff;
            const double pw = pow(por, -dragGamma);
            for (int d = 0; d < c.nd; d++) fd[d] = c.drag_scale * (sc * dv[d] * pw);
        }
        for (int d = 0; d < c.nd; d++) {
            fdrag_out[d] = (c.dem_vol / ma) * (fv[d] + fpfb[d]) + (c.dens / ma) * fd[d];
            f[d] += fdrag_out[d];
        }
    } else {
        for (int d = 0; d < c.nd; d++) fvel[d] *= 1.0;  /* unnormalised, as the reference leaves it */
    }
    for (int d = 0; d < 3; d++) {
        s.row(FD_FVEL + d)[a] = fvel[d];
        s.row(FD_FDRAG + d)[a] = fdrag_out[d];
    }
    s.row(FD_POR)[a] = por;
    s.row(FD_SHEP)[a] = sum;
    /* calcDEMContacts over the DEM buckets (sph.h:1676-1706, LINEAR) */
    const double Ra = radius_of(c, s, (int)a);
    const CellCoord cd = dem_cell_of(c, ra);
    scan_cells(cd, c.ddims, c.periodic, c.nd, start, gi.n_sph_cells, [&](int b, const int *sh) {
        if (b == a && !(sh[0] | sh[1] | sh[2])) return;
        if (s.irow(FI_IAM)[b] != T_DEM) return;
        double dx[3], r2;
        if (!pair_geom(c, s, b, sh, ra, ha, dx, r2)) return;
        const double r = sqrt(r2);
        double nrm[3] = {0, 0, 0}, dv[3] = {0, 0, 0};
        for (int d = 0; d < c.nd; d++) {
            nrm[d] = dx[d] / r;
            dv[d] = va[d] - s.row(FD_VHAT + d)[b];
        }
        const double overlap = (Ra + radius_of(c, s, b)) - r;
        if (overlap > 0) {
            const double od = -dot3(dv, nrm, c.nd);
            const double sN = c.dem_k * overlap + c.dem_gamma * od;
            for (int d = 0; d < c.nd; d++) {
                const double fN = (sN * nrm[d]) / ma;
                fpv[d] += fN;
                f[d] += fN;
            }
        }
    });
    for (int d = 0; d < c.nd; d++) {
        s.row(FD_F + d)[a] = f[d];
        s.row(FD_FP + d)[a] = fpv[d];
    }
}

}  // namespace

void zero_dem_shep(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "zero_dem_shep", k_zero_dem_shep, grid_for(c->n, 256), 256, 0, c->A, c->n);
}
void run_porosity(sphdem_ctx *c) {
    if (c->f64_dem) {
        if (!c->only_dem) couple64(c, 0);
        return;
    }
    zero_dem_shep(c);
    SPHDEM_LAUNCH(c, "porosity_fp64", k_porosity, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->buf.start, c->g, c->n);
}
void run_dem_drag(sphdem_ctx *c) {
    if (c->f64_dem) {
        if (!c->only_dem) couple64(c, 1);
        return;
    }
    SPHDEM_LAUNCH(c, "dem_drag_fp64", k_dem_drag, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->buf.start, c->g, c->n);
}
void run_eos(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "eos_fp64", k_eos, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->n);
}
void run_dem_accel(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "dem_accel", k_dem_accel, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_dem_end(sphdem_ctx *c) {
    if (c->f64_dem) {
        dem_end64(c, !c->only_dem);
        return;
    }
    SPHDEM_LAUNCH(c, "dem_end_fp64", k_dem_end, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->buf.start, c->g, c->n);
}

}  // namespace sphdem
