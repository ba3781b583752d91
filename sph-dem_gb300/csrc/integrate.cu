/*
 * Elementwise parts of a step: the integrator functors of sphIncompress.h
 * (driftR 620-641, driftRAndKick 643-676, driftRest 678-704, kick 706-742,
 * initSumsMiddle 744-763, initSumsEnd 765-767), the dt choice of
 * sphIncompress.cpp:126-154, and the device built-ins of the case hooks
 * (gravity, planar DEM walls and DEM freezing in the pattern of
 * sediment3D/customSim.cpp:5-113).
 *
 * Each launch fuses every per-particle functor the reference runs back to
 * back in one phase, so a phase touches each live field once; a whole step
 * fuses further, across the phases and into the rebuild that follows
 * (k_sweep in binning.cu).  All of them are HBM-bound: bytes per particle =
 * the rows read + written in elementwise.cuh.
 */
#include "elementwise.cuh"

namespace sphdem {
namespace {

constexpr int BLK = 256;

__global__ void k_globals_op(DevCfg c, DevGlobals *g, int op) {
    if (threadIdx.x || blockIdx.x) return;
    switch (op) {
        case OP_MIDDLE_BEGIN:
            g->new_dt = g->maxdt;
            g->new_dt_bits = dbits(g->maxdt);
            break;
        case OP_SET_DT: {
            double nd = __longlong_as_double((long long)g->new_dt_bits);
            if (c.liq_dem()) {
                nd = fmin(nd, c.liq_dem_timestep);
                if (g->time > c.time_drop) nd = fmin(nd, c.dem_timestep);
            }
            g->new_dt = nd;
            g->old_dt = g->dt;
            if (c.flags & SPHDEM_F_FIXED_DT) g->dt = g->maxdt;
            else g->dt = nd;
            break;
        }
        case OP_END_BEGIN:
            g->dem_dt = g->maxdt;
            break;
        case OP_STEP_INC:
            g->step += 1;
            break;
    }
}

/* DEM_BLOCK: calcAvForce over the DEM particles (sphIncompress.h:107-110) and
 * the mean (sphIncompress.cpp:232-236).  One block, a fixed reduction tree:
 * the same sum on every run. */
constexpr int AVF_BLK = 1024;
__global__ void __launch_bounds__(AVF_BLK) k_dem_block(DevCfg c, DevState s, DevGlobals *g, int64_t n) {
    __shared__ double sh[4][AVF_BLK / 32];
    double acc[4] = {0, 0, 0, 0};
    for (int64_t i = threadIdx.x; i < n; i += AVF_BLK) {
        if (s.irow(FI_IAM)[i] != T_DEM) continue;
        for (int d = 0; d < c.nd; d++) acc[d] += s.row(FD_F + d)[i];
        acc[3] += 1.0;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int k = 0; k < 4; k++) {
        double v = acc[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh[k][w] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[4] = {0, 0, 0, 0};
        for (int k = 0; k < 4; k++)
            for (int j = 0; j < AVF_BLK / 32; j++) t[k] += sh[k][j];
        for (int d = 0; d < 3; d++) g->dem_avf[d] = t[3] > 0 ? t[d] / t[3] : 0.0;
    }
}

/* one elementwise phase on its own (the phase-level calls) */
enum Phase : int { PH_START = 0, PH_HOOK_MIDDLE, PH_MIDDLE_TAIL, PH_HOOK_END, PH_END_DRIFT, PH_END_TAIL, PH_HOOK_AFTER };
template <int PH>
__global__ void k_phase(DevCfg c, DevState s, DevGlobals *g, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const double dt = g->dt;
    if (i == 0) {
        if (PH == PH_START || PH == PH_END_DRIFT) g->time = g->time + dt / 2;
        if (PH == PH_END_DRIFT && c.liq_dem()) g->dem_dt = g->maxdt;
    }
    if (i >= n) return;
    const int t = s.irow(FI_IAM)[i];
    if (PH == PH_START) start_particle(c, s, i, t, dt);
    if (PH == PH_HOOK_MIDDLE) hook_before_middle_particle(c, s, i, t);
    if (PH == PH_MIDDLE_TAIL) middle_tail_particle(c, s, i, t, dt, g->old_dt, g->time);
    if (PH == PH_HOOK_END) hook_before_end_particle(c, s, i, t, g->time);
    if (PH == PH_END_DRIFT) end_drift_particle(c, s, i, t, dt);
    if (PH == PH_END_TAIL) end_tail_particle(c, s, g, i, t, dt, g->time);
    if (PH == PH_HOOK_AFTER) freeze_particle(c, s, i, t, g->time);
}

/* end() tail and the afterEnd hook, of a whole step */
__global__ void k_end_tail(DevCfg c, DevState s, DevGlobals *g, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = s.irow(FI_IAM)[i];
    end_tail_particle(c, s, g, i, t, g->dt, g->time);
    freeze_particle(c, s, i, t, g->time);
}

__global__ void k_h_derived(DevCfg c, DevState s, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.irow(FI_IAM)[i] == T_DEAD) return;
    h_derived(c, s, i);
}

}  // namespace

void run_h_derived(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "h_derived", k_h_derived, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->n);
}

void globals_op(sphdem_ctx *c, int op) {
    SPHDEM_LAUNCH(c, "globals_op", k_globals_op, 1, 32, 0, c->cfg, c->g, op);
}
void run_start(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "start", k_phase<PH_START>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_hook_before_middle(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "hook_before_middle", k_phase<PH_HOOK_MIDDLE>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_middle_tail(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "middle_tail", k_phase<PH_MIDDLE_TAIL>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_end_drift(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "end_drift", k_phase<PH_END_DRIFT>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_dem_block(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "dem_block", k_dem_block, 1, AVF_BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_end_tail(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "end_tail", k_phase<PH_END_TAIL>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_step_tail(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "end_tail", k_end_tail, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_hook_before_end(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "hook_before_end", k_phase<PH_HOOK_END>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}
void run_hook_after_end(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "hook_after_end", k_phase<PH_HOOK_AFTER>, grid_for(c->n, BLK), BLK, 0, c->cfg, c->A, c->g, c->n);
}

}  // namespace sphdem
