/*
 * Per-particle parts of a step, as device functions: the integrator functors of
 * sphIncompress.h and the built-in case hooks.  t is the particle's type.
 */
#pragma once

#include "internal.cuh"

namespace sphdem {
namespace {

__device__ __forceinline__ void eos(const DevCfg &c, const DevState &s, int64_t i) {
    const double dens = s.row(FD_DENS)[i];
    double press;
    if (c.liq_dem()) {
        const double x = dens * recip(c, c.refd * s.row(FD_POR)[i]);
        double xg;
        if (c.gamma == 7.0) {
            const double x2 = x * x;
            xg = x2 * x2 * x2 * x;
        } else {
            xg = pow(x, c.gamma);
        }
        press = c.prb * (xg - 1.0);
    } else {
        const double x = dens / c.refd;
        const double x2 = x * x;
        press = c.prb * (x2 * x2 * x2 * x - 1.0);
    }
    const double rd = recip(c, dens);
    s.row(FD_PRESS)[i] = press;
    s.row(FD_PDR2)[i] = press * (rd * rd);
}

/* start(): driftRAndKick + driftRest + initSumsMiddle for sph/sphBoundary,
 * driftR for dem (sphIncompress.cpp:3-38, no density re-init) */
__device__ __forceinline__ void start_particle(const DevCfg &c, const DevState &s, int64_t i, int t, double dt) {
    const double hd = dt / 2;
    if (is_sph_or_sphb(t)) {
        for (int d = 0; d < c.nd; d++) {
            double *r = s.row(FD_R + d), *vh = s.row(FD_VHAT + d);
            r[i] += hd * vh[i];
            if (t != T_SPHB) {
                double *v = s.row(FD_V + d), *f = s.row(FD_F + d);
                s.row(FD_V0 + d)[i] = v[i];
                s.row(FD_VHAT0 + d)[i] = vh[i];
                v[i] += hd * f[i];
                vh[i] += hd * f[i];
            }
        }
        double *dens = s.row(FD_DENS);
        dens[i] += hd * s.row(FD_DDDT)[i];
        if (!(c.flags & SPHDEM_F_CONST_H)) {
            s.row(FD_H)[i] = smoothing_length(c, s.row(FD_MASS)[i] * recip(c, dens[i]));
            h_derived(c, s, i);
        }
        for (int d = 0; d < 3; d++) {
            s.row(FD_F + d)[i] = 0.0;
            s.row(FD_FP + d)[i] = 0.0;
            s.row(FD_FV + d)[i] = 0.0;
            s.row(FD_FB + d)[i] = 0.0;
        }
    } else if (c.liq_dem() && t == T_DEM) {
        for (int d = 0; d < c.nd; d++) s.row(FD_R + d)[i] += hd * s.row(FD_VHAT + d)[i];
    }
}

/* beforeMiddle built-in: gravity on type sph (sediment3D/customSim.cpp:90-95) */
__device__ __forceinline__ void hook_before_middle_particle(const DevCfg &c, const DevState &s, int64_t i, int t) {
    if (t != T_SPH) return;
    for (int d = 0; d < c.nd; d++)
        if (c.g_sph[d] != 0.0) s.row(FD_F + d)[i] += c.g_sph[d];
}

/* the time step of the middle phase (sphIncompress.cpp:126-154) from the
 * smallest bound of its passes */
__device__ __forceinline__ double choose_dt(const DevCfg &c, const DevGlobals *g, double *new_dt) {
    double nd = __longlong_as_double((long long)g->new_dt_bits);
    if (c.liq_dem()) {
        nd = fmin(nd, c.liq_dem_timestep);
        if (g->time > c.time_drop) nd = fmin(nd, c.dem_timestep);
    }
    *new_dt = nd;
    return c.flags & SPHDEM_F_FIXED_DT ? g->maxdt : nd;
}

/* middle() after the force loop: kick sph/sphBoundary with (oldDt+dt)/2,
 * initSumsEnd, then for dem driftRAndKick + initSumsMiddle
 * (sphIncompress.cpp:157-164) */
__device__ __forceinline__ void middle_tail_particle(const DevCfg &c, const DevState &s, int64_t i, int t, double dt,
                                                     double old_dt, double time) {
    if (is_sph_or_sphb(t)) {
        if (t == T_SPH) {
            const double k = 0.5 * old_dt + 0.5 * dt;
            const bool damp = time < c.damptime;
            for (int d = 0; d < c.nd; d++) {
                const double f = s.row(FD_F + d)[i];
                double v = s.row(FD_V0 + d)[i] + k * f;
                double vh = s.row(FD_VHAT0 + d)[i] + k * f;
                if (damp) {
                    v *= 0.98;
                    vh *= 0.98;
                }
                s.row(FD_V + d)[i] = v;
                s.row(FD_VHAT + d)[i] = vh;
            }
        }
        s.row(FD_DDDT)[i] = 0.0;
    } else if (c.liq_dem() && t == T_DEM) {
        const double hd = dt / 2;
        for (int d = 0; d < c.nd; d++) {
            double *r = s.row(FD_R + d), *v = s.row(FD_V + d), *vh = s.row(FD_VHAT + d);
            const double f = s.row(FD_F + d)[i];
            r[i] += hd * vh[i];
            s.row(FD_V0 + d)[i] = v[i];
            s.row(FD_VHAT0 + d)[i] = vh[i];
            v[i] += hd * f;
            vh[i] += hd * f;
        }
        for (int d = 0; d < 3; d++) {
            s.row(FD_F + d)[i] = 0.0;
            s.row(FD_FP + d)[i] = 0.0;
            s.row(FD_FV + d)[i] = 0.0;
            s.row(FD_FB + d)[i] = 0.0;
        }
    }
}

/* end(): driftR for sph/sphBoundary (sphIncompress.cpp:169-183) */
__device__ __forceinline__ void end_drift_particle(const DevCfg &c, const DevState &s, int64_t i, int t, double dt) {
    if (!is_sph_or_sphb(t)) return;
    for (int d = 0; d < c.nd; d++) s.row(FD_R + d)[i] += (dt / 2) * s.row(FD_VHAT + d)[i];
}

/* end() tail: dem kick(dt/2,dt/2) (sphIncompress.cpp:239), driftRest for
 * sph/sphBoundary (245) and calcEnergies (249, sphIncompress.h:769-781): EOS
 * refresh, elastic energy u += dt pdr2 dddt, and for sph the viscous energy
 * eViscF += dt (-vhat . fv) */
__device__ __forceinline__ void end_tail_particle(const DevCfg &c, const DevState &s, const DevGlobals *g, int64_t i, int t,
                                                  double dt, double time) {
    if (c.liq_dem() && t == T_DEM) {
        const double k = 0.5 * dt + 0.5 * dt;
        const bool damp = time < c.damptime;
        const bool block = c.flags & SPHDEM_F_DEM_BLOCK;
        for (int d = 0; d < c.nd; d++) {
            if (block) s.row(FD_F + d)[i] = g->dem_avf[d];   /* setAvForce, sphIncompress.h:112-114 */
            const double f = s.row(FD_F + d)[i];
            double v = s.row(FD_V0 + d)[i] + k * f;
            double vh = s.row(FD_VHAT0 + d)[i] + k * f;
            if (damp) {
                v *= 0.98;
                vh *= 0.98;
            }
            s.row(FD_V + d)[i] = v;
            s.row(FD_VHAT + d)[i] = vh;
        }
    } else if (is_sph_or_sphb(t)) {
        double *dens = s.row(FD_DENS);
        dens[i] += (dt / 2) * s.row(FD_DDDT)[i];
        if (!(c.flags & SPHDEM_F_CONST_H)) {
            s.row(FD_H)[i] = smoothing_length(c, s.row(FD_MASS)[i] * recip(c, dens[i]));
            h_derived(c, s, i);
        }
        eos(c, s, i);
        const double dudt = s.row(FD_PDR2)[i] * s.row(FD_DDDT)[i];
        s.row(FD_DUDT)[i] = dudt;
        s.row(FD_U)[i] += dt * dudt;
        if (t == T_SPH) {
            double w = 0.0;
            for (int d = 0; d < c.nd; d++) w += s.row(FD_VHAT + d)[i] * s.row(FD_FV + d)[i];
            s.row(FD_DEVISCF)[i] = -w;
            s.row(FD_EVISCF)[i] += dt * (-w);
        }
    }
}

/* DEM at rest until the freeze ends */
__device__ __forceinline__ void freeze_particle(const DevCfg &c, const DevState &s, int64_t i, int t, double time) {
    if (!c.liq_dem() || t != T_DEM || !(time <= c.freeze_until)) return;
    for (int d = 0; d < 3; d++) {
        s.row(FD_F + d)[i] = 0.0;
        s.row(FD_V + d)[i] = 0.0;
        s.row(FD_VHAT + d)[i] = 0.0;
    }
}

/* beforeEnd built-ins for dem: gravity, planar walls, freeze */
__device__ __forceinline__ void hook_before_end_particle(const DevCfg &c, const DevState &s, int64_t i, int t, double time) {
    if (!c.liq_dem() || t != T_DEM) return;
    const double R = s.row(FD_RADIUS)[i] > 0.0 ? s.row(FD_RADIUS)[i] : c.dem_radius;
    double rr[3] = {0, 0, 0}, vv[3] = {0, 0, 0}, f[3] = {0, 0, 0}, fb[3] = {0, 0, 0};
    for (int d = 0; d < c.nd; d++) {
        rr[d] = s.row(FD_R + d)[i];
        vv[d] = s.row(FD_VHAT + d)[i];
        f[d] = s.row(FD_F + d)[i];
        fb[d] = s.row(FD_FB + d)[i];
        if (c.g_dem[d] != 0.0) f[d] += c.g_dem[d];
    }
    for (int w = 0; w < c.n_walls; w++) {
        const double *wn = c.wall_n[w];
        double dd[3] = {0, 0, 0};
        for (int d = 0; d < c.nd; d++) dd[d] = rr[d] - c.wall_p[w][d];
        const double dist = c.nd == 3 ? dd[0] * wn[0] + (dd[1] * wn[1] + dd[2] * wn[2]) : dd[0] * wn[0] + dd[1] * wn[1];
        const double overlap = R - dist;
        if (overlap > 0.0) {
            const double vn = c.nd == 3 ? vv[0] * wn[0] + (vv[1] * wn[1] + vv[2] * wn[2]) : vv[0] * wn[0] + vv[1] * wn[1];
            const double sN = c.dem_k * overlap + c.dem_gamma * (-vn), m = s.row(FD_MASS)[i];
            for (int d = 0; d < c.nd; d++) {
                if (wn[d] == 0.0) continue; /* an FP64 division */
                const double fN = (sN * wn[d]) / m;
                fb[d] += fN;
                f[d] += fN;
            }
        }
    }
    for (int d = 0; d < c.nd; d++) {
        s.row(FD_F + d)[i] = f[d];
        s.row(FD_FB + d)[i] = fb[d];
    }
    freeze_particle(c, s, i, t, time);
}

}  // namespace
}  // namespace sphdem
