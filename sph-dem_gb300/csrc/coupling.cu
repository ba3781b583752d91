/*
 * SPH-DEM coupling and DEM contact passes, in the handle's precision (R = float
 * on mixed handles, double on FP64 ones):
 *   k_couple<.., 0>  calcPorosity + calcShepSum       sph.h:1323-1341, 1303-1320
 *   k_couple<.., 1>  calcDEMtoSPHDrag + finalisePorosity + setPorosityForBoundary
 *                                                     sph.h:1343-1362, 1289-1296, 1263-1265
 *   k_fpi            calcFPI's sums                   sph.h:1708-1792
 *   k_dem_finish     calcFPI's normalisation, Di Felice drag, calcDEMContacts
 *                                                     sph.h:1575-1631, 1676-1706
 *
 * One in six to one in thirty of the candidates of a bucket stencil takes part,
 * so each pass searches and computes in turn: the search runs in FP32 on bucket
 * offsets (with the proven band, inside which the reference's FP64 predicate
 * decides) and appends the partners it finds to a shared-memory queue; the pair
 * arithmetic then takes the queue's entries with all lanes busy.  That matters
 * most for FP64 arithmetic, which the chip does on two lanes per SM whether
 * one or all lanes of the warp take part.
 *
 * Neighbour sets are the reference's: coupling partners within Rc by its
 * asymmetric bucket rule (dataLL.cpp:1154-1190), FPI partners and contacts by
 * its neighbour predicate, periodic images only where it holds a ghost.
 *
 * All are bound by the search: latency of the bucket records below ~100,000
 * particles, instruction issue above.  Before / now, us: 1.08 M particles (mixed)
 * porosity 530 / 438, drag 328 / 94, FPI and contacts 571 / 385; 69,758 (FP64)
 * 1,303 / 188, 1,155 / 42, 3,737 / 134; contacts of 50,000 settling spheres (FP64)
 * 515 / 68.
 */
#include <algorithm>

#include "fp64.cuh"
#include "mixed.cuh"

namespace sphdem {
namespace {

constexpr int CQ = 16; /* queued partners per thread of the coupling passes */


__device__ __forceinline__ void shift_of(int shp, int *sh) {
    sh[0] = (shp & 3) - 1;
    sh[1] = ((shp >> 2) & 3) - 1;
    sh[2] = ((shp >> 4) & 3) - 1;
}

/* FP64 displacement r_a - image(r_b) */
template <int ND>
__device__ __forceinline__ void pair_dx(const DevCfg &c, const DevState &s, const double *ra, int b, int shp, double *dx) {
    int sh[3];
    shift_of(shp, sh);
#pragma unroll
    for (int d = 0; d < ND; d++) dx[d] = dsub(ra[d], image_pos(s.row(FD_R + d)[b], sh[d], c.rmin[d], c.rmax[d]));
}

/* one warp-aggregated atomic reserves k entries per lane of cnt; every lane
 * of the warp calls it; returns this lane's first entry */
__device__ __forceinline__ int64_t tap_reserve(int k, int *cnt) {
    const int lane = threadIdx.x & 31;
    int incl = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    int base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(cnt, total);
    base = __shfl_sync(0xffffffffu, base, 31);
    return (int64_t)base + incl - k;
}

/* Does SPH bucket cs list DEM bucket cd (dataLL.cpp:1154-1190)? lim_ceil =
 * ceil(couple_lim): for the integer sums rP < couple_lim <=> rP < lim_ceil */
template <int ND>
__device__ __forceinline__ bool bucket_rule(const int *cs, const int *cd, int num, int lim_ceil) {
    int rP = 0, rM = 0;
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const int o = cd[d] - cs[d];
        if (o < -num || o > num) return false;
        rP += (o + 1) * (o + 1);
        rM += (o - 1) * (o - 1);
    }
    return ND == 1 || rP < lim_ceil || rM < lim_ceil;
}

/* a compensated sum in FP32, a plain one in FP64 */
template <typename R>
struct Sum {
    Kahan k;
    __device__ __forceinline__ void init() { k.init(0.f); }
    __device__ __forceinline__ void add(float x) { k.add(x); }
    __device__ __forceinline__ double value() const { return k.s; }
};
template <>
struct Sum<double> {
    double s;
    __device__ __forceinline__ void init() { s = 0.0; }
    __device__ __forceinline__ void add(double x) { s += x; }
    __device__ __forceinline__ double value() const { return s; }
};

/* G threads per fluid particle: partners among the DEM particles of the 3^d DEM
 * buckets around it (DEM buckets are at least Rc wide), each thread in its share
 * of the bucket columns.  The search keeps to positions; bucket rule and image
 * are looked up for the queued candidates only.  TAP (adjoint replay
 * only): the pairs go to the tap table tt of step *tslot -- mode 0 counts them
 * and reserves the particle's entries, mode 1 (the same pairs) writes them. */
/* Mode 0 keeps its pairs and their kernel values for mode 1, which runs at the
 * same positions and would find them again by the same search (an eighth of the
 * time goes into the pairs, the rest into the search): entry k of thread t at
 * [k * threads + t], kept_pairs(G) of them; num counts them all, and a thread with
 * more searches again. */
template <typename R>
struct Kept {
    int *id, *num;
    R *w;
    int64_t threads;
};
template <int ND, int MODE, typename R, bool TAP, int G>
__global__ void __launch_bounds__(BLK) k_couple(DevCfg c, const DevCfg *__restrict__ cp, DevState s,
                                                const int *__restrict__ start, const int *__restrict__ skey,
                                                const DevGlobals *__restrict__ g, const float4 *__restrict__ P0,
                                                const float4 *__restrict__ P1, const float4 *__restrict__ P2,
                                                const float4 *__restrict__ DP, const int *__restrict__ tg,
                                                Kept<R> keep, TapTable tt, const int *__restrict__ tslot,
                                                int64_t n_all) {
    constexpr int Z = ND - 1;
    constexpr int NCOL = Z == 2 ? 9 : (Z == 1 ? 3 : 1);
    constexpr bool F64 = sizeof(R) == 8;
    /* displacement (FP32) and DEM particle | image code << 26 of queued partners */
    __shared__ float4 s_hit[CQ][BLK];
    const int nsc = g->n_sph_cells, n_t = start[nsc];
    const int64_t a = (blockIdx.x * (int64_t)BLK + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    if (blockIdx.x * (int64_t)(BLK / G) >= n_t) return;
    const int ta = a < n_t ? (tg[a] & 0xff) : -1;
    const bool act = is_sph_or_sphb(ta);
    if (MODE == 1 && is_boundary(ta)) s.row(FD_POR)[a] = 1.0;
    const int64_t thread = a * G + sub;
    constexpr int LIMIT = kept_pairs(G);
    /* this thread's pairs: counted (mode 0), known (mode 1), -1 without kept pairs */
    int num = 0;
    if (MODE == 1) num = keep.num ? (act ? keep.num[thread] : 0) : -1;
    int ntap = 0, js = 0;
    int *tout = nullptr;
    if (TAP) {
        js = *tslot;
        if (MODE == 1) {
            /* the particle's entries, its threads' one after the other */
            int before = num;
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, before, o, G);
                if (sub >= o) before += v;
            }
            if (act) {
                const int2 o = tt.oc[(int64_t)js * n_all + s.irow(FI_TAG)[a]];
                /* a particle whose entries overflowed the table recorded none */
                if (o.y > 0) tout = tt.nb + (int64_t)js * tt.cap + o.x + (before - num);
            }
        }
    }
    Sum<R> por, dpd, acc[ND];
    por.init();
    dpd.init();
#pragma unroll
    for (int k = 0; k < ND; k++) acc[k].init();
    /* DEM -> fluid drag of one pair with kernel value W */
    auto drag = [&](int b, R W, R rdens) {
        if constexpr (F64) {
            const double sc = s.row(FD_MASS)[b] * rdens * W * rcp_pos(s.row(FD_SHEP)[b]);
#pragma unroll
            for (int k = 0; k < ND; k++) acc[k].add(-sc * s.row(FD_FDRAG + k)[b]);
        } else {
            const float4 x = DP[b]; /* (m / shep, fdrag) */
            const float sc = x.x * rdens * W, f[3] = {x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < ND; k++) acc[k].add(-sc * f[k]);
        }
    };
    auto tap = [&](int id) {
        if (tout && ntap < num) tout[ntap] = s.irow(FI_TAG)[id & B_MASK] | (id & ~B_MASK);
        ntap++;
    };
    const R densa = !act ? (R)1 : (F64 ? (R)s.row(FD_DENS)[a] : (R)P2[a].x);
    const R rdens = ND == 2 ? (R)(1.0 / (2.0 * c.dem_radius)) / densa : (R)1 / densa;
    const bool search = act && (MODE == 0 || num < 0 || num > LIMIT);
    for (int k = 0; MODE == 1 && !search && k < num; k++) {
        const int64_t at = k * keep.threads + thread;
        const int id = keep.id[at];
        if (TAP) tap(id);
        drag(id & B_MASK, keep.w[at], rdens);
    }
    if (__any_sync(0xffffffffu, search)) {
        double ra[3] = {0, 0, 0};
        int cs[3] = {0, 0, 0};
        float off[3] = {0.f, 0.f, 0.f}, dcf[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < ND; d++) {
            if (act) {
                ra[d] = s.row(FD_R + d)[a];
                cs[d] = ref_dem_cell(ra[d], c, d);
            }
            dcf[d] = (float)c.dcell[d];
        }
        const CellCoord cc = dem_cell_of(c, ra);
        float lmax = 0.f;
#pragma unroll
        for (int d = 0; d < ND; d++) {
            off[d] = (float)(ra[d] - dem_origin(c, d, cc.c[d]));
            lmax = fmaxf(lmax, fabsf(off[d]) + 2.f * dcf[d]);
        }
        const float rc2 = (float)c.rc2, band = fp32_band(rc2, lmax * lmax);
        const int lim_ceil = (int)ceil(c.couple_lim);
        const float wconf = (float)c.wcon;
        R va[3] = {0, 0, 0};
        if (MODE == 0 && act) {
            if (F64) {
#pragma unroll
                for (int d = 0; d < ND; d++) va[d] = s.row(FD_VHAT + d)[a];
            } else {
                const float4 v = P1[a];
                va[0] = v.x;
                va[1] = v.y;
                va[2] = v.z;
            }
        }
        const R dvol = !act ? (R)0 : (F64 ? (R)(s.row(FD_MASS)[a] / densa) : (R)(P1[a].w / (float)densa));
        const R two_over_rc = (R)c.two_over_rc;
        /* one partner's terms */
        auto pair = [&](float4 h) {
            const int id = __float_as_int(h.w), b = id & B_MASK, shp = (unsigned)id >> B_BITS;
            R d[3] = {(R)h.x, (R)h.y, (R)h.z}, r2, r;
            int sh[3], cd[3] = {0, 0, 0};
            shift_of(shp, sh);
#pragma unroll
            for (int k = 0; k < ND; k++)
                cd[k] = sh[k] ? ref_dem_cell(image_pos(s.row(FD_R + k)[b], sh[k], c.rmin[k], c.rmax[k]), c, k)
                              : s.irow(FI_RDC0 + k)[b];
            if (!bucket_rule<ND>(cs, cd, c.couple_num, lim_ceil)) return;
            if (shp != 0x15 && !img_ok<ND>(tg[b] >> 8, sh)) return;
            if constexpr (F64) {
                pair_dx<ND>(c, s, ra, b, shp, d);
                r2 = exact_len2(d, ND);
                if (!(r2 < c.rc2)) return; /* decided in FP64 */
                r = sqrt_pos(r2);
            } else {
                r2 = d[0] * d[0];
#pragma unroll
                for (int k = 1; k < ND; k++) r2 = fmaf(d[k], d[k], r2);
                if (r2 >= rc2 - band && !exact_pair<ND>(cp, s, (int)a, b, sh[0], sh[1], sh[2], c.rc2, 1)) return;
                r = sqrtf(r2);
            }
            if (TAP && MODE == 1) tap(id);
            const R q = r * two_over_rc;
            R W, t3;
            if constexpr (F64) {
                const double t = positive_part(2.0 - q);
                t3 = t * t * t;
                W = c.c_ihn * (c.wcon * (t3 * t) * fma(2.0, q, 1.0));
            } else {
                const float t = fmaxf(2.f - q, 0.f);
                t3 = t * t * t;
                W = (float)c.c_ihn * (wconf * (t3 * t) * (1.f + 2.f * q));
            }
            if (MODE == 0) {
                if (keep.num && num < LIMIT) {
                    keep.id[num * keep.threads + thread] = id;
                    keep.w[num * keep.threads + thread] = W;
                }
                num++;
                por.add((R)c.por_incr * W);
                /* the gradient factor dK/dq / q of the coupling kernel; a pair at r = 0 has none (dx = 0) */
                const R Fq = (R)(-10.0 * c.wcon * c.c_ihn2 * c.dem_vol) * t3;
                R vd = 0;
                if constexpr (F64) {
#pragma unroll
                    for (int k = 0; k < ND; k++) vd = fma(va[k] - s.row(FD_VHAT + k)[b], d[k], vd);
                } else {
                    const float4 x = P1[b];
                    vd = (va[0] - x.x) * d[0];
                    if (ND > 1) vd += (va[1] - x.y) * d[1];
                    if (ND > 2) vd += (va[2] - x.z) * d[2];
                }
                dpd.add(-(vd * Fq));
#pragma unroll
                for (int k = 0; k < ND; k++) acc[k].add(d[k] * Fq);
                atomicAdd(&s.row(FD_SHEP)[b], (double)(dvol * W));
            } else {
                drag(b, W, rdens);
            }
        };
        /* the warp goes through the columns together, every thread in its own
         * range, and takes the queued candidates together when a queue is full */
        const float reach2 = rc2 + band;
        int qn = 0;
        auto drain = [&]() {
            for (int k = 0; __any_sync(0xffffffffu, k < qn); k++)
                if (k < qn) pair(s_hit[k][threadIdx.x]);
            qn = 0;
        };
#pragma unroll 1
        for (int c0 = 0; c0 < NCOL; c0 += G) {
            const int col = c0 + sub;
            /* columns of buckets out of reach on the leading axes */
            float far2 = 0.f;
            if (Z > 0) {
                const int o0 = Z == 2 ? col / 3 - 1 : col - 1;
                const float f0 = o0 < 0 ? off[0] : (o0 > 0 ? dcf[0] - off[0] : 0.f);
                far2 = fmaxf(f0, 0.f) * fmaxf(f0, 0.f);
            }
            if (Z > 1) {
                const int o1 = col % 3 - 1;
                const float f1 = o1 < 0 ? off[1] : (o1 > 0 ? dcf[1] - off[1] : 0.f);
                far2 += fmaxf(f1, 0.f) * fmaxf(f1, 0.f);
            }
            const bool near = search && col < NCOL && far2 * (1.f - 1e-5f) <= reach2;
#pragma unroll 1
            for (int piece = c.periodic[Z] ? 0 : 1; piece < (c.periodic[Z] ? 3 : 2); piece++) {
                RangeEntry re = {0, 0, 0, 0, 0x15, 0, 0.f, 0.f};
                if (near) re = range_entry<ND>(3 * col + piece, cc.c, cc.c[Z], cc.c[Z], c.ddims, c.periodic, dcf, nsc, start);
                int b = re.b0;
                const int end = re.b0 + re.cnt;
                /* the next candidate's record in flight */
                float4 pn = make_float4(0.f, 0.f, 0.f, 0.f);
                int kn = 0;
                if (b < end) {
                    pn = P0[b];
                    kn = skey[b];
                }
                const float ox = Z > 0 ? off[0] - re.ox : off[0], oy = Z > 1 ? off[1] - re.oy : off[1];
                while (__any_sync(0xffffffffu, b < end)) {
                    if (b < end) {
                        const float4 pb = pn;
                        const float zb = (float)(re.zoff + (kn - re.lin)) * dcf[Z];
                        const int bb = b++;
                        if (b < end) {
                            pn = P0[b];
                            kn = skey[b];
                        }
                        float d[3] = {ox - pb.x, ND > 1 ? oy - pb.y : 0.f, ND > 2 ? off[2] - pb.z : 0.f};
                        d[Z] -= zb;
                        float r2 = d[0] * d[0];
                        if (ND > 1) r2 = fmaf(d[1], d[1], r2);
                        if (ND > 2) r2 = fmaf(d[2], d[2], r2);
                        if (r2 < reach2)
                            s_hit[qn++][threadIdx.x] = make_float4(d[0], d[1], d[2], __int_as_float(bb | (re.shp << B_BITS)));
                    }
                    if (__any_sync(0xffffffffu, qn == CQ)) drain();
                }
            }
        }
        drain();
    }
    if (MODE == 0 && act && keep.num) keep.num[thread] = num;
    if (TAP && MODE == 0) {
        const int64_t o = tap_reserve(num, tt.cnt + js);
        int all = num;
#pragma unroll
        for (int k = 1; k < G; k <<= 1) all += __shfl_xor_sync(0xffffffffu, all, k);
        if (act && sub == 0) tt.oc[(int64_t)js * n_all + s.irow(FI_TAG)[a]] = make_int2((int)o, o + all <= tt.cap ? all : 0);
    }
    double vp = por.value(), vd = dpd.value(), vs[ND];
    if (MODE == 0) {
        vp = lane_sum<G>(vp);
        vd = lane_sum<G>(vd);
    }
#pragma unroll
    for (int k = 0; k < ND; k++) vs[k] = lane_sum<G>(acc[k].value());
    if (!act || sub) return;
    if (MODE == 0) {
        s.row(FD_POR)[a] = vp;
        s.row(FD_DPORDT)[a] = vd;
#pragma unroll
        for (int k = 0; k < ND; k++) s.row(FD_GPOR + k)[a] = vs[k];
    } else {
#pragma unroll
        for (int k = 0; k < ND; k++) {
            const double v = vs[k];
            s.row(FD_FDRAG + k)[a] = v;
            s.row(FD_F + k)[a] += v;
        }
        double p = 1.0 - s.row(FD_POR)[a];
        if (p < 0.37) {
            p = 0.37;
            s.row(FD_DPORDT)[a] = 0.0;
            for (int k = 0; k < 3; k++) s.row(FD_GPOR + k)[a] = 0.0;
        }
        s.row(FD_POR)[a] = p;
    }
}

/* (m/shep, fdrag) of every DEM particle for the DEM->SPH drag (sph.h:1359) */
__global__ void k_pack_dem_drag(DevState s, const float4 *__restrict__ P1, float4 *__restrict__ DP, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.irow(FI_IAM)[i] != T_DEM) return;
    const float sh = (float)s.row(FD_SHEP)[i];
    DP[i] = make_float4(sh != 0.f ? P1[i].w / sh : 0.f, (float)s.row(FD_FDRAG)[i], (float)s.row(FD_FDRAG + 1)[i],
                        (float)s.row(FD_FDRAG + 2)[i]);
}

/* fields the DEM side gathers from fluid neighbours in calcFPI (sph.h:1708-1792):
 * Q0 = (fp+fb, fv.x), Q1 = (fv.y, fv.z) */
__global__ void k_pack_fpi(DevState s, float4 *__restrict__ Q0, float2 *__restrict__ Q1, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f[3];
#pragma unroll
    for (int d = 0; d < 3; d++) f[d] = (float)(s.row(FD_FP + d)[i] + s.row(FD_FB + d)[i]);
    Q0[i] = make_float4(f[0], f[1], f[2], (float)s.row(FD_FV)[i]);
    Q1[i] = make_float2((float)s.row(FD_FV + 1)[i], (float)s.row(FD_FV + 2)[i]);
}

/* exclusive prefix of v over the warp; *total = the sum */
__device__ __forceinline__ int warp_excl_scan(int v, int lane, int *total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    *total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

/* the lane whose range holds flat index j: the last lane with excl <= j */
__device__ __forceinline__ int warp_range_src(int excl, int j) {
    int src = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int e = __shfl_sync(0xffffffffu, excl, src + step);
        if (e <= j) src += step;
    }
    return src;
}

/* sums of 16 values over the warp in 16 additions per lane: lane l ends with
 * value (l >> 1 & 15, bits reversed by halves): each step sends half of the
 * values and keeps the other half */
template <typename R>
__device__ __forceinline__ R warp_sum16(R *v, int lane) {
#pragma unroll
    for (int o = 16, half = 8; half >= 1; o >>= 1, half >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const R keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

/* calcFPI's sums, one warp per DEM particle.  Candidates of the 3^d SPH buckets
 * come from a range table (one lane per bucket run) and are spread flat over the
 * lanes; a lane queues its partners and the warp takes one of each lane at a
 * time.  (A queue of the warp instead, taken 32 partners at a time, runs at full
 * lanes but adds in another order, and the partial sums of a particle at rest in
 * a swarm under drag cancel: its path over 10 steps moved by up to 2e-9 of the box.)
 * The unnormalised sums go
 * to the particle's fvel, porosity and Shepard rows and, where calcFPI normalises
 * (Shepard sum > 0.5), its fb and fv rows.  TAP: the partners of DEM particle w
 * of the DEM range also go to slots w * per .. of table tf of step *tslot. */
constexpr int FPI_QUEUE = 8;
template <int ND, typename R, bool TAP>
__global__ void __launch_bounds__(BLK) k_fpi(DevCfg c, const DevCfg *__restrict__ cp, DevState s,
                                             const int *__restrict__ start, const int *__restrict__ skey,
                                             const DevGlobals *__restrict__ g, const float4 *__restrict__ P0,
                                             const float4 *__restrict__ P1, const float4 *__restrict__ P2,
                                             const float4 *__restrict__ Q0, const float2 *__restrict__ Q1,
                                             const int *__restrict__ tg, const float4 *__restrict__ DS, TapTable tf,
                                             const int *__restrict__ tslot, int64_t n_all) {
    constexpr int Z = ND - 1;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr bool F64 = sizeof(R) == 8;
    __shared__ int s_queue[FPI_QUEUE][BLK];
    const int lane = threadIdx.x & 31;
    const int warps = (blockDim.x >> 5) * gridDim.x;
    const int nsc = g->n_sph_cells;
    const int dem0 = start[nsc], dem1 = start[nsc + c.n_dem_cells];
    const int sdims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    float cell[3], cs2 = 0.f;
    load_cell32(c, g, cell);
#pragma unroll
    for (int d = 0; d < ND; d++) cs2 = fmaxf(cs2, 4.f * cell[d] * cell[d]);
    const float wcon = (float)c.wcon;
    for (int a = dem0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); a < dem1; a += warps) {
        const float ha = P0[a].w;
        const float4 ds = DS[a];
        int cs[3] = {0, 0, 0}, kf = 0, js = 0;
        int *fout = nullptr;
        if (TAP) {
            js = *tslot;
            const int64_t w = a - dem0;
            if ((w + 1) * tf.per <= tf.cap) fout = tf.nb + (int64_t)js * tf.cap + w * tf.per;
        }
        decode<ND>(__float_as_int(ds.w), sdims, cs);
        const float oa[3] = {ds.x, ds.y, ds.z};
        double ra[3] = {0, 0, 0};
        if (F64)
#pragma unroll
            for (int d = 0; d < ND; d++) ra[d] = s.row(FD_R + d)[a];
        /* fp + fb, fv, vel: 3 each; porosity; Shepard sum */
        R v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = 0;
        int qn = 0;
        /* the terms of the queued partners */
        auto take = [&]() {
            for (int t = 0; __any_sync(FULL, t < qn); t++) {
                if (TAP) {
                    const unsigned m = __ballot_sync(FULL, t < qn);
                    const int at = kf + __popc(m & ((1u << lane) - 1u));
                    if (t < qn && fout && at < tf.per) {
                        const int id = s_queue[t][threadIdx.x];
                        fout[at] = s.irow(FI_TAG)[id & B_MASK] | (id & ~B_MASK);
                    }
                    kf += __popc(m);
                }
                if (t >= qn) continue;
                const int id = s_queue[t][threadIdx.x], b = id & B_MASK, shp = (unsigned)id >> B_BITS;
                if constexpr (F64) {
                    double d[3] = {0, 0, 0};
                    pair_dx<ND>(c, s, ra, b, shp, d);
                    double r2 = d[0] * d[0];
#pragma unroll
                    for (int k = 1; k < ND; k++) r2 = fma(d[k], d[k], r2);
                    const double q = sqrt_pos(r2) * s.row(FD_IH)[b], t = positive_part(2.0 - q), t2 = t * t;
                    const double mb = s.row(FD_MASS)[b];
                    const double mW = mb * (s.row(FD_IHN)[b] * (c.wcon * (t2 * t2) * fma(2.0, q, 1.0)));
                    const double dvW = mW * rcp_pos(s.row(FD_DENS)[b]);
#pragma unroll
                    for (int k = 0; k < ND; k++) {
                        v[k] = fma(mW, s.row(FD_FP + k)[b] + s.row(FD_FB + k)[b], v[k]);
                        v[3 + k] = fma(mW + dvW, s.row(FD_FV + k)[b], v[3 + k]);
                        v[6 + k] = fma(dvW, s.row(FD_VHAT + k)[b], v[6 + k]);
                    }
                    v[9] = fma(dvW, s.row(FD_POR)[b], v[9]);
                    v[10] += dvW;
                } else {
                    const float4 pb = P0[b], vb = P1[b], xb = P2[b], q0 = Q0[b];
                    const float2 q1 = Q1[b];
                    /* the displacement again, from the partner's bucket */
                    int cb[3] = {0, 0, 0}, sh[3];
                    decode<ND>(skey[b], sdims, cb);
                    shift_of(shp, sh);
                    const float qb[3] = {pb.x, pb.y, pb.z};
                    float r2 = 0.f;
#pragma unroll
                    for (int k = 0; k < ND; k++) {
                        const float d = oa[k] - (qb[k] + (float)(cb[k] + sh[k] * sdims[k] - cs[k]) * cell[k]);
                        r2 = fmaf(d, d, r2);
                    }
                    const float mb = fabsf(vb.w), q = sqrtf(r2) * xb.w;
                    const float Wab = powi<ND>(xb.w) * wK32(q, wcon);
                    const float dvW = (mb / xb.x) * Wab, mW = mb * Wab;
                    const float fb[3] = {q0.x, q0.y, q0.z}, fv[3] = {q0.w, q1.x, q1.y}, vel[3] = {vb.x, vb.y, vb.z};
#pragma unroll
                    for (int k = 0; k < ND; k++) {
                        v[k] += mW * fb[k];
                        v[3 + k] += mW * fv[k] + dvW * fv[k];
                        v[6 + k] += dvW * vel[k];
                    }
                    v[9] += dvW * xb.z;
                    v[10] += dvW;
                }
            }
            qn = 0;
        };
        const RangeEntry re = range_entry<ND>(lane, cs, cs[Z], cs[Z], sdims, c.periodic, cell, 0, start);
        int total = 0;
        const int excl = warp_excl_scan(re.cnt, lane, &total);
        for (int t = 0; t < total; t += 32) {
            const int j = t + lane;
            const int src = warp_range_src(excl, j);
            const int b0 = __shfl_sync(FULL, re.b0, src), ex = __shfl_sync(FULL, excl, src);
            const int lin = __shfl_sync(FULL, re.lin, src), zoff = __shfl_sync(FULL, re.zoff, src);
            const int shp = __shfl_sync(FULL, re.shp, src);
            const float ox = __shfl_sync(FULL, re.ox, src), oy = __shfl_sync(FULL, re.oy, src);
            bool hit = j < total;
            const int b = b0 + (hit ? j - ex : 0);
            if (hit) {
                const float4 pb = P0[b];
                float q[3] = {pb.x, pb.y, pb.z};
                if (Z > 0) q[0] += ox;
                if (Z > 1) q[1] += oy;
                q[Z] += (float)(zoff + (skey[b] - lin)) * cell[Z];
                float r2 = 0.f;
#pragma unroll
                for (int k = 0; k < ND; k++) r2 = fmaf(oa[k] - q[k], oa[k] - q[k], r2);
                const float tt = 2.f * fmaxf(ha, pb.w), T = tt * tt;
                const float band = fp32_band(T, cs2);
                hit = r2 <= T + band;
                if (hit) {
                    int sh[3];
                    shift_of(shp, sh);
                    const int tgb = tg[b];
                    hit = (tgb & 0xff) != T_BOUNDARY && (shp == 0x15 || img_ok<ND>(tgb >> 8, sh)) &&
                          (r2 < T - band || exact_pair<ND>(cp, s, a, b, sh[0], sh[1], sh[2], 0.0, 0));
                }
            }
            if (hit) s_queue[qn++][threadIdx.x] = b | (shp << B_BITS);
            if (__any_sync(FULL, qn == FPI_QUEUE)) take();
        }
        take();
        if (TAP && lane == 0) {
            const int64_t w = a - dem0, at = (int64_t)js * n_all + s.irow(FI_TAG)[a];
            tf.oc[at] = make_int2((int)(w * tf.per), fout && kf <= tf.per ? kf : 0);
            if (!fout || kf > tf.per) atomicMax(tf.cnt + js, (int)tf.cap + 1); /* marks the step overflowed */
        }
        const R x = warp_sum16(v, lane);
        const int k = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
        const R sum = __shfl_sync(FULL, x, 20); /* value 10 */
        if ((lane & 1) == 0 && k <= 10) {
            if (k < 6) {
                const int d = k % 3;
                if (d < ND && sum > (R)0.5) s.row((k < 3 ? FD_FB : FD_FV) + d)[a] = x;
            } else if (k < 9) {
                s.row(FD_FVEL + k - 6)[a] = x;
            } else {
                s.row(k == 9 ? FD_POR : FD_SHEP)[a] = x;
            }
        }
    }
}

/* calcFPI's normalisation and the Di Felice drag from the sums of k_fpi, in R;
 * adds the drag to f */
template <int ND, typename R>
__device__ __forceinline__ void fpi_drag(const DevCfg &c, const DevState &s, int64_t a, double *f) {
    const R sum = (R)s.row(FD_SHEP)[a];
    if (!(sum > (R)0.5)) {
        for (int k = 0; k < 3; k++) s.row(FD_FDRAG + k)[a] = 0.0;
        return;
    }
    const R rsum = (R)1 / sum;
    const R pr = (R)s.row(FD_POR)[a] * rsum;
    R fvfp[3] = {0, 0, 0}, dv[3] = {0, 0, 0}, vd2 = 0;
#pragma unroll
    for (int k = 0; k < ND; k++) {
        const R fb = (R)s.row(FD_FB + k)[a] * rsum, fv = (R)s.row(FD_FV + k)[a] * rsum, vel = (R)s.row(FD_FVEL + k)[a] * rsum;
        s.row(FD_FB + k)[a] = fb;
        s.row(FD_FV + k)[a] = fv;
        s.row(FD_FVEL + k)[a] = vel;
        fvfp[k] = fv + fb;
        dv[k] = pr * (vel - (R)s.row(FD_VHAT + k)[a]);
        vd2 += dv[k] * dv[k];
    }
    s.row(FD_POR)[a] = pr;
    /* calcParticleDrag, Di Felice (sph.h:1575-1631) */
    R fd[3] = {0, 0, 0};
    if (vd2 != 0) {
        if constexpr (sizeof(R) == 8) {
            const double vdiff = sqrt(vd2), A = c.pi * (c.dem_radius * c.dem_radius);
            const double Re = (2.0 * c.dem_radius / c.viscosity) * vdiff, lg = 1.5 - log10(Re);
            const double dragGamma = 3.7 - 0.65 * exp(-(lg * lg) / 2.0), cc0 = 0.63 + 4.8 / sqrt(Re);
            const double sc = (1.0 / 2.0) * A * (cc0 * cc0) * vdiff, pw = pow(pr, -dragGamma);
            for (int d = 0; d < ND; d++) fd[d] = c.drag_scale * (sc * dv[d] * pw);
        } else {
            const float vdiff = sqrtf(vd2), A = (float)(c.pi * (c.dem_radius * c.dem_radius));
            const float Re = (float)(2.0 * c.dem_radius / c.viscosity) * vdiff, lg = 1.5f - log10f(Re);
            const float dragGamma = 3.7f - 0.65f * expf(-(lg * lg) / 2.f), cc0 = 0.63f + 4.8f / sqrtf(Re);
            const float sc = 0.5f * A * (cc0 * cc0) * vdiff, pw = powf(pr, -dragGamma) * (float)c.drag_scale;
            for (int d = 0; d < ND; d++) fd[d] = sc * dv[d] * pw;
        }
    }
    const double ma = s.row(FD_MASS)[a];
    const R vm = (R)(c.dem_vol / ma), dm = (R)(c.dens / ma);
    for (int k = 0; k < 3; k++) {
        const R drag = k < ND ? vm * fvfp[k] + dm * fd[k] : (R)0;
        s.row(FD_FDRAG + k)[a] = drag;
        if (k < ND) f[k] += drag;
    }
}

/* DEM contacts (calcDEMContacts, sph.h:1676-1706, LINEAR), FP64 as the overlap
 * (Ra + Rb) - r cancels, and the end of calcFPI.  Four lanes share a DEM
 * particle: each searches its share of the bucket columns in FP32 for spheres
 * that may touch and queues them; the queued contacts are then taken in step.
 * TAP: the touching contacts of DEM particle w of the DEM range also go to
 * slots w * per .. of table tct of step *tslot. */
constexpr int CT_LANES = 4;
constexpr int CT_QUEUE = 8;
template <int ND, typename R, bool TAP>
__global__ void __launch_bounds__(BLK) k_dem_finish(DevCfg c, DevState s, const int *__restrict__ start,
                                                    const int *__restrict__ skey, const DevGlobals *__restrict__ g,
                                                    const float4 *__restrict__ P0, const int *__restrict__ tg, int fluid,
                                                    TapTable tct, const int *__restrict__ tslot, int64_t n_all) {
    constexpr int Z = ND - 1;
    constexpr int NCOL = Z == 2 ? 9 : (Z == 1 ? 3 : 1);
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ int s_queue[CT_QUEUE][BLK];
    const int lane = threadIdx.x & 31, sub = threadIdx.x % CT_LANES;
    const unsigned group = ((1u << CT_LANES) - 1u) << (lane - sub);
    const int nsc = g->n_sph_cells;
    const int dem0 = start[nsc], dem1 = start[nsc + c.n_dem_cells];
    float cell[3], cd2 = 0.f, cmax = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        cell[d] = (float)c.dcell[d];
        if (d < ND) {
            cd2 = fmaxf(cd2, 4.f * cell[d] * cell[d]);
            cmax = fmaxf(cmax, cell[d]);
        }
    }
    const int per_pass = gridDim.x * (BLK / CT_LANES);
    for (int w0 = blockIdx.x * (BLK / CT_LANES) + (threadIdx.x >> 5) * (32 / CT_LANES); dem0 + w0 < dem1; w0 += per_pass) {
        const int a = dem0 + w0 + lane / CT_LANES;
        const bool act = a < dem1;
        int js = 0, kc = 0;
        int *cout = nullptr;
        if (TAP) {
            js = *tslot;
            const int64_t w = a - dem0;
            if (act && (w + 1) * tct.per <= tct.cap) cout = tct.nb + (int64_t)js * tct.cap + w * tct.per;
        }
        double ra[3] = {0, 0, 0}, va[3] = {0, 0, 0}, fc[3] = {0, 0, 0}, Ra = 0.0, ha = 0.0, rma = 0.0;
        int qn = 0, col = sub, piece = -1, b = 0, end = 0, lin = 0, zoff = 0, shp = 0x15;
        float ox = 0.f, oy = 0.f, oa[3] = {0.f, 0.f, 0.f}, haf = 0.f, Raf = 0.f;
        int cc[3] = {0, 0, 0};
        if (act) {
#pragma unroll
            for (int d = 0; d < ND; d++) {
                ra[d] = s.row(FD_R + d)[a];
                va[d] = s.row(FD_VHAT + d)[a];
            }
            Ra = s.row(FD_RADIUS)[a] > 0 ? s.row(FD_RADIUS)[a] : c.dem_radius;
            ha = s.row(FD_H)[a];
            rma = 1.0 / s.row(FD_MASS)[a];
            const float4 pa = P0[a];
            oa[0] = pa.x;
            oa[1] = pa.y;
            oa[2] = pa.z;
            haf = pa.w;
            Raf = (float)Ra;
            decode<ND>(skey[a] - nsc, c.ddims, cc);
        }
        bool more = act && col < NCOL;
        while (__any_sync(FULL, more)) {
            /* search until the queue is full or the columns are done */
            while (more && qn < CT_QUEUE) {
                if (b >= end) {
                    /* the next range: period pieces of the column, then the lane's next column */
                    const int last = c.periodic[Z] ? 2 : 1;
                    piece = piece < 0 ? (c.periodic[Z] ? 0 : 1) : piece + 1;
                    if (piece > last) {
                        col += CT_LANES;
                        piece = c.periodic[Z] ? 0 : 1;
                    }
                    if (col >= NCOL) {
                        more = false;
                        break;
                    }
                    const RangeEntry re = range_entry<ND>(3 * col + piece, cc, cc[Z], cc[Z], c.ddims, c.periodic, cell, nsc, start);
                    b = re.b0;
                    end = re.b0 + re.cnt;
                    lin = re.lin;
                    zoff = re.zoff;
                    shp = re.shp;
                    ox = re.ox;
                    oy = re.oy;
                    continue;
                }
                const int bb = b++;
                if (bb == a && shp == 0x15) continue;
                const float4 pb = P0[bb];
                float q[3] = {pb.x, pb.y, pb.z};
                if (Z > 0) q[0] += ox;
                if (Z > 1) q[1] += oy;
                q[Z] += (float)(zoff + (skey[bb] - lin)) * cell[Z];
                float r2 = 0.f;
#pragma unroll
                for (int k = 0; k < ND; k++) r2 = fmaf(oa[k] - q[k], oa[k] - q[k], r2);
                const float tt = 2.f * fmaxf(haf, pb.w), T = tt * tt;
                if (r2 > T + fp32_band(T, cd2)) continue;
                const double Rb = s.row(FD_RADIUS)[bb] > 0 ? s.row(FD_RADIUS)[bb] : c.dem_radius;
                const float touch = (Raf + (float)Rb) * 1.0001f + 2e-6f * cmax;
                if (r2 > touch * touch) continue;
                s_queue[qn++][threadIdx.x] = bb | (shp << B_BITS);
            }
            /* the queued contacts, one per lane at a time */
            for (int k = 0; __any_sync(FULL, k < qn); k++) {
                bool touching = false;
                int id = 0;
                if (k < qn) {
                    id = s_queue[k][threadIdx.x];
                    const int bb = id & B_MASK, sp = (unsigned)id >> B_BITS;
                    double dx[3] = {0, 0, 0};
                    pair_dx<ND>(c, s, ra, bb, sp, dx);
                    const double r2 = exact_len2(dx, ND);
                    /* r^2 <= (2 max h)^2: five FP32 roundings are below 4e-7, so FP32 decides
                     * unless the two are nearly equal */
                    const float hm = fmaxf(haf, P0[bb].w), r2f = (float)r2, T = 4.f * hm * hm;
                    const bool fits = T > 1e-30f;
                    bool near = fits && r2f < T * (1.f - 1e-6f);
                    if (!near && !(fits && r2f > T * (1.f + 1e-6f))) {
                        const double hb = s.row(FD_H)[bb], t = 2.0 * (ha > hb ? ha : hb);
                        near = r2 <= dmul(t, t);
                    }
                    int sh[3];
                    shift_of(sp, sh);
                    if (near && (sp == 0x15 || img_ok<ND>(tg[bb] >> 8, sh))) {
                        /* the overlap is a difference of r and the radii, and shows the last
                         * place of r: with the root to 0.75 ulp the paths of 50,000
                         * settling spheres were off by 2.1e-13, with 0.5 ulp by 1.7e-13 */
                        double ri;
                        const double r = sqrt_pos<true>(r2, &ri);
                        const double Rb = s.row(FD_RADIUS)[bb] > 0 ? s.row(FD_RADIUS)[bb] : c.dem_radius;
                        const double overlap = (Ra + Rb) - r;
                        if (overlap > 0) {
                            touching = true;
                            double vn = 0.0;
#pragma unroll
                            for (int d = 0; d < ND; d++) vn = fma(va[d] - s.row(FD_VHAT + d)[bb], dx[d], vn);
                            /* normal dx / r, approach speed -vn / r */
                            const double sN = fma(c.dem_k, overlap, -c.dem_gamma * (vn * ri)) * ri * rma;
#pragma unroll
                            for (int d = 0; d < ND; d++) fc[d] = fma(sN, dx[d], fc[d]);
                        }
                    }
                }
                if (TAP) {
                    const unsigned m = __ballot_sync(FULL, touching) & group;
                    const int at = kc + __popc(m & ((1u << lane) - 1u));
                    if (touching && cout && at < tct.per) cout[at] = s.irow(FI_TAG)[id & B_MASK] | (id & ~B_MASK);
                    kc += __popc(m);
                }
            }
            qn = 0;
        }
#pragma unroll
        for (int d = 0; d < ND; d++)
#pragma unroll
            for (int o = 1; o < CT_LANES; o <<= 1) fc[d] += __shfl_xor_sync(FULL, fc[d], o);
        if (!act || sub) continue;
        if (TAP) {
            const int64_t w = a - dem0, at = (int64_t)js * n_all + s.irow(FI_TAG)[a];
            tct.oc[at] = make_int2((int)(w * tct.per), cout && kc <= tct.per ? kc : 0);
            if (!cout || kc > tct.per) atomicMax(tct.cnt + js, (int)tct.cap + 1);
        }
        double f[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < ND; d++) f[d] = s.row(FD_F + d)[a];
        if (fluid) {
            fpi_drag<ND, R>(c, s, a, f);
        } else {
            for (int d = 0; d < 3; d++) s.row(FD_FVEL + d)[a] = s.row(FD_FDRAG + d)[a] = 0.0;
            s.row(FD_POR)[a] = 0.0;
            s.row(FD_SHEP)[a] = 0.0;
        }
#pragma unroll
        for (int d = 0; d < ND; d++) {
            s.row(FD_F + d)[a] = f[d] + fc[d];
            s.row(FD_FP + d)[a] += fc[d];
        }
    }
}

/* blocks of a grid-stride pass: enough for `threads`, at most one wave of resident blocks */
template <auto K>
int wave_blocks(int64_t threads) {
    static int resident = 0;
    if (!resident) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, BLK, 0);
        resident = std::max(1, sms * per_sm);
    }
    return (int)std::max<int64_t>(1, std::min<int64_t>(resident, (threads + BLK - 1) / BLK));
}

template <int MODE, typename R>
void couple(sphdem_ctx *c, const char *name) {
    const TapTable tt = c->tap ? c->tap->cpl : TapTable{};
    const int *ts = c->tap ? c->tap->slot : nullptr;
    /* four threads per particle while one leaves the chip short of warps; both
     * passes, us with 1 / 4: FP32 3.8k 116 / 68, 23k 131 / 87, 91k 159 / 175; FP64
     * 3.8k 208 / 110, 23k 243 / 197, 70k 353 / 337 (before the kept pairs) */
    const bool split = c->n < CP_SPLIT_BELOW;
    const Kept<R> keep = {c->cp_id, c->cp_num, reinterpret_cast<R *>(c->cp_w), c->n * (split ? 4 : 1)};
#define LK_(ND, T, G)                                                                                             \
    SPHDEM_LAUNCH(c, name, (k_couple<ND, MODE, R, T, G>), grid_for(c->n * G, BLK), BLK, 0, c->cfg, c->dcfg, c->A,   \
                  c->buf.start, c->buf.skey, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_dp, c->mx_tg, keep, tt, ts,     \
                  c->n)
#define L_(ND)                                        \
    do {                                              \
        if constexpr (sizeof(R) == 4) {               \
            if (c->tap) {                             \
                if (split)                            \
                    LK_(ND, true, 4);                 \
                else                                  \
                    LK_(ND, true, 1);                 \
                break;                                \
            }                                         \
        }                                             \
        if (split)                                    \
            LK_(ND, false, 4);                        \
        else                                          \
            LK_(ND, false, 1);                        \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LK_
}

template <typename R>
void dem_end_passes(sphdem_ctx *c, bool fluid) {
    const TapTable tf = c->tap ? c->tap->fpi : TapTable{}, tct = c->tap ? c->tap->ct : TapTable{};
    const int *ts = c->tap ? c->tap->slot : nullptr;
    const char *fpi_name = sizeof(R) == 4 ? "fpi32" : "fpi_fp64", *end_name = sizeof(R) == 4 ? "dem_end32" : "dem_end_fp64";
#define LK_(ND, T)                                                                                                  \
    do {                                                                                                            \
        if (fluid)                                                                                                  \
            SPHDEM_LAUNCH(c, fpi_name, (k_fpi<ND, R, T>), (wave_blocks<k_fpi<ND, R, T>>(c->n * 32)), BLK, 0, c->cfg,    \
                          c->dcfg, c->A, c->buf.start, c->buf.skey, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_q0,    \
                          c->mx_q1, c->mx_tg, c->mx_ds, tf, ts, c->n);                                               \
        SPHDEM_LAUNCH(c, end_name, (k_dem_finish<ND, R, T>), (wave_blocks<k_dem_finish<ND, R, T>>(c->n * CT_LANES)), \
                      BLK, 0, c->cfg, c->A, c->buf.start, c->buf.skey, c->g, c->mx_pos, c->mx_tg, (int)fluid, tct, ts, \
                      c->n);                                                                                         \
    } while (0)
#define L_(ND)                                        \
    do {                                              \
        if constexpr (sizeof(R) == 4) {               \
            if (c->tap) {                             \
                LK_(ND, true);                        \
                break;                                \
            }                                         \
        }                                             \
        LK_(ND, false);                               \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LK_
}

}  // namespace

/* the FP64 passes on FP32 searches (handles with the records) */
void couple64(sphdem_ctx *c, int mode) {
    if (mode == 0) couple<0, double>(c, "porosity_fp64");
    else couple<1, double>(c, "dem_drag_fp64");
}
void dem_end64(sphdem_ctx *c, bool fluid) { dem_end_passes<double>(c, fluid); }

namespace mixed {

void porosity(sphdem_ctx *c) { couple<0, float>(c, "porosity32"); }

void dem_drag(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "pack_dem_drag32", k_pack_dem_drag, grid_for(c->n, 256), 256, 0, c->A, c->mx_vel, c->mx_dp, c->n);
    couple<1, float>(c, "dem_drag32");
}

void dem_end(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "pack_fpi32", k_pack_fpi, grid_for(c->n, 256), 256, 0, c->A, c->mx_q0, c->mx_q1, c->n);
    dem_end_passes<float>(c, true);
}

}  // namespace mixed
}  // namespace sphdem
