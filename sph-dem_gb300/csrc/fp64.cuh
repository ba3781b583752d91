/*
 * Device helpers of the FP64 pair passes: the Wendland kernel, the exact
 * neighbour predicate and the time-step reduction.
 */
#pragma once

#include <cfloat>

#include "internal.cuh"
#include "series.cuh"

namespace sphdem {
namespace {

__device__ __forceinline__ double dot3(const double *a, const double *b, int nd) {
    if (nd == 3) return a[0] * b[0] + (a[1] * b[1] + a[2] * b[2]);
    if (nd == 2) return a[0] * b[0] + a[1] * b[1];
    return a[0] * b[0];
}

/* Wendland C2 pieces (sph.h:74-80, 136-142, 199-205): K and dK/dq */
__device__ __forceinline__ double wK(double q, double wcon) {
    if (q > 2.0) return 0.0;
    const double t = 2.0 - q, t2 = t * t;
    return wcon * (t2 * t2) * (1.0 + 2.0 * q);
}
__device__ __forceinline__ double wdK(double q, double wcon) {
    if (q > 2.0) return 0.0;
    const double t = 2.0 - q, t2 = t * t;
    return wcon * (-4 * (t2 * t) * (1 + 2 * q) + 2 * (t2 * t2));
}

/* the displacement r_a - image(r_b) and the exact neighbour predicate */
__device__ __forceinline__ bool pair_geom(const DevCfg &c, const DevState &s, int b, const int *sh,
                                          const double *ra, double ha, double *dx, double &r2) {
    for (int d = 0; d < 3; d++) dx[d] = 0.0;
    for (int d = 0; d < c.nd; d++)
        dx[d] = dsub(ra[d], image_pos(s.row(FD_R + d)[b], sh[d], c.rmin[d], c.rmax[d]));
    r2 = exact_len2(dx, c.nd);
    const double hb = s.row(FD_H)[b];
    const double t = 2.0 * (ha > hb ? ha : hb);
    if (r2 > dmul(t, t)) return false;
    if ((sh[0] | sh[1] | sh[2]) && !image_exists(s.irow(FI_GCODE)[b], sh, c.nd)) return false;
    return true;
}

__device__ __forceinline__ void block_min_atomic(double v, unsigned long long *target) {
    __shared__ double smin[32];
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) smin[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? smin[lane] : DBL_MAX;
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v < DBL_MAX) atomic_min_pos(target, v);
    }
}

/* 1/x for x > 0 (rcp_series) */
__device__ __forceinline__ double rcp_pos(double x) {
    const float xf = (float)x;
    if (!(xf > 1e-30f && xf < 1e30f)) return 1.0 / x;
    float yf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
    return rcp_series(x, (double)yf);
}

/* sqrt(x) and, where asked, 1/sqrt(x) of x >= 0 (sqrt_series; FULL: sqrt_series_full) */
template <bool FULL = false>
__device__ __forceinline__ double sqrt_pos(double x, double *inv = nullptr) {
    const float xf = (float)x;
    if (!(xf > 1e-30f && xf < 1e30f)) {
        const double r = sqrt(x);
        if (inv) *inv = r > 0.0 ? 1.0 / r : 0.0;
        return r;
    }
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
    if (FULL) return sqrt_series_full(x, (double)yf, inv);
    return sqrt_series(x, (double)yf, inv);
}

/* max(x, 0) by the sign bit (an integer operation) */
__device__ __forceinline__ double positive_part(double x) {
    return __double_as_longlong(x) < 0 ? 0.0 : x;
}

/* the smaller of two non-negative doubles by their bit patterns */
__device__ __forceinline__ double min_pos(double a, double b) {
    return __double_as_longlong(a) < __double_as_longlong(b) ? a : b;
}

template <int G>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace
}  // namespace sphdem
