/*
 * Device helpers shared by the mixed-precision pair passes: FP32 kernel
 * values and compensated sums, bucket keys and neighbour-list tiles, the
 * repulsive boundary force and the staging of neighbour records in shared
 * memory.
 */
#pragma once

#include <cfloat>
#include <climits>

#include "internal.cuh"
#include "series.cuh"

namespace sphdem {
namespace {

constexpr int BLK = 128;
constexpr int B_BITS = 26;
constexpr int B_MASK = (1 << B_BITS) - 1;

/* a + b = r + e, e the rounding error */
__device__ __forceinline__ void two_sum(float a, float b, float &r, float &e) {
    r = a + b;
    const float bb = r - a;
    e = (a - (r - bb)) + (b - bb);
}

/* the sum of t + c over G consecutive lanes, c a small correction of t */
template <int G>
__device__ __forceinline__ float join_lanes(float t, float c) {
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const float to = __shfl_xor_sync(0xffffffffu, t, o), co = __shfl_xor_sync(0xffffffffu, c, o);
        float u, e;
        two_sum(t, to, u, e);
        t = u;
        c = (c + co) + e;
    }
    return t + c;
}

struct Kahan {
    float s, c;
    __device__ __forceinline__ void init(float v) {
        s = v;
        c = 0.f;
    }
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    /* the total of G consecutive lanes' sums (all lanes of the warp call it) with
     * the additions' rounding errors kept */
    template <int G>
    __device__ __forceinline__ float total() const {
        return join_lanes<G>(s, -c);
    }
};

/* A plain FP32 sum with the same interface, for sums whose rounding does
 * not reach the results' tolerance: the calcOmega sum under
 * VAR_H_CORRECTION, where Omega = 1 + h sum / (rho NDIM) is an O(1) factor
 * known to ~1e-6 from ~100 terms. */
struct Plain {
    float s;
    __device__ __forceinline__ void init(float v) { s = v; }
    __device__ __forceinline__ void add(float x) { s += x; }
};

/* Two Kahan sums side by side in packed FP32 (n: the negated compensations) */
struct Kahan2 {
    float2 s, n;
    __device__ __forceinline__ void init() { s = n = make_float2(0.f, 0.f); }
    /* adds a * b; the product is not rounded by itself */
    __device__ __forceinline__ void add_product(float2 a, float2 b) {
        const float2 neg = make_float2(-1.f, -1.f);
        const float2 y = __ffma2_rn(a, b, n);
        const float2 t = __fadd2_rn(s, y);
        n = __ffma2_rn(__ffma2_rn(s, neg, t), neg, y);
        s = t;
    }
    /* the total of both sums and of G consecutive lanes' (all lanes of the
     * warp call it); the additions' rounding errors are kept */
    template <int G>
    __device__ __forceinline__ float total() const {
        float t, e;
        two_sum(s.x, s.y, t, e);
        return join_lanes<G>(t, e + (n.x + n.y));
    }
};

__device__ __forceinline__ float wK32(float q, float wcon) {
    if (q > 2.f) return 0.f;
    const float t = 2.f - q, t2 = t * t;
    return wcon * (t2 * t2) * (1.f + 2.f * q);
}
__device__ __forceinline__ float wdK32(float q, float wcon) {
    if (q > 2.f) return 0.f;
    const float t = 2.f - q, t2 = t * t;
    return wcon * (-4.f * (t2 * t) * (1.f + 2.f * q) + 2.f * (t2 * t2));
}

template <int ND>
__device__ __forceinline__ float powi(float x) {
    float r = x;
#pragma unroll
    for (int k = 1; k < ND; k++) r *= x;
    return r;
}

template <int ND>
__device__ __forceinline__ void decode(int key, const int *dims, int *cc) {
    if (ND == 3) {
        cc[2] = key % dims[2];
        key /= dims[2];
        cc[1] = key % dims[1];
        cc[0] = key / dims[1];
    } else if (ND == 2) {
        cc[1] = key % dims[1];
        cc[0] = key / dims[1];
    } else {
        cc[0] = key;
    }
}

__device__ __forceinline__ int code_stride(int d) { return d == 0 ? 9 : (d == 1 ? 3 : 1); }

__device__ __forceinline__ void nl_decode_code(int code, int *o) {
    o[0] = code / 9 - 1;
    o[1] = (code / 3) % 3 - 1;
    o[2] = code % 3 - 1;
}

/* FP64 origin of SPH bucket `cell` on axis d */
__device__ __forceinline__ double sph_origin(const DevCfg &c, const DevGlobals *g, int d, int cell) {
    return c.periodic[d] ? c.dmin[d] + cell * g->scell[d] : c.dmin[d] + (cell - 3) * g->sr2;
}

__device__ __forceinline__ double dem_origin(const DevCfg &c, int d, int cell) {
    return c.dorig[d] + cell * c.dcell[d];
}


template <int ND>
__device__ __forceinline__ bool img_ok(int gcode, const int *sh) {
#pragma unroll
    for (int d = 0; d < ND; d++) {
        if (sh[d] == 0) continue;
        const int ic = (gcode >> (2 * d)) & 3;
        if (sh[d] < 0 ? ic != 2 : ic != 0) return false;
    }
    return true;
}

/* The reference's FP64 predicate for a pair inside the FP32 band. */
template <int ND>
__device__ __noinline__ bool exact_pair(const DevCfg *__restrict__ cp, const DevState s, int a, int b, int sh0,
                                        int sh1, int sh2, double lim2, int strict) {
    const int sh[3] = {sh0, sh1, sh2};
    double dx[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < ND; d++)
        dx[d] = dsub(s.row(FD_R + d)[a], image_pos(s.row(FD_R + d)[b], sh[d], cp->rmin[d], cp->rmax[d]));
    const double r2 = exact_len2(dx, ND);
    if (lim2 > 0) return strict ? r2 < lim2 : r2 <= lim2;
    const double ha = s.row(FD_H)[a], hb = s.row(FD_H)[b];
    const double t = 2.0 * (ha > hb ? ha : hb);
    return r2 <= dmul(t, t);
}

/* Half-width of the band around a cut-off T = R^2 inside which an FP32 r^2
 * built from bucket offsets cannot decide: each displacement component is
 * off by < 6 * 2^-24 L when L bounds the magnitudes of the offset terms, so
 * r^2 by < 1.25e-6 L max(L, R) + 1.8e-7 r^2, and T by < 1.8e-7 T. */
__device__ __forceinline__ float fp32_band(float T, float L2) { return fmaf(5e-7f, T, 1.5e-6f * fmaxf(L2, T)); }

/* One lane's entry of a bucket range table around a run of buckets (ccol
 * on the leading axes, zmin..zmax on the last axis Z): lane = 3 * column +
 * period piece, for the 3^(d-1) neighbour columns; each entry is a run of
 * consecutive keys key0 + lin .. (buckets zmin-1 .. zmax+1 of the column,
 * cut at a periodic seam).  Entries of other lanes are empty. */
struct RangeEntry {
    int b0, cnt, lin, zoff, shp, code;
    float ox, oy;
};

template <int ND>
__device__ __forceinline__ RangeEntry range_entry(int lane, const int *ccol, int zmin, int zmax, const int *dims,
                                                  const int *periodic, const float *cell, int key0,
                                                  const int *__restrict__ start) {
    constexpr int Z = ND - 1;
    constexpr int NCOL = Z == 2 ? 9 : (Z == 1 ? 3 : 1);
    RangeEntry r = {0, 0, 0, 0, 0x15, 0, 0.f, 0.f};
    if (lane >= 3 * NCOL) return r;
    const int colidx = lane / 3, wz = lane % 3 - 1;
    int o[2] = {0, 0};
    if (Z == 2) {
        o[0] = colidx / 3 - 1;
        o[1] = colidx % 3 - 1;
    } else if (Z == 1) {
        o[0] = colidx - 1;
    }
    bool ok = wz == 0 || periodic[Z];
    int col_lin = 0, code = 0, shp = 0;
    float off[2] = {0.f, 0.f};
#pragma unroll
    for (int d = ND; d < 3; d++) {
        shp |= 1 << (2 * d);
        code += code_stride(d);
    }
#pragma unroll
    for (int d = 0; d < Z; d++) {
        int t = ccol[d] + o[d], shd = 0;
        if (t < 0) {
            ok = ok && periodic[d];
            t += dims[d];
            shd = -1;
        } else if (t >= dims[d]) {
            ok = ok && periodic[d];
            t -= dims[d];
            shd = 1;
        }
        col_lin = col_lin * dims[d] + t;
        code += (o[d] + 1) * code_stride(d);
        off[d] = (float)o[d] * cell[d];
        shp |= (shd + 1) << (2 * d);
    }
    shp |= (wz + 1) << (2 * Z);
    const int zdim = dims[Z];
    const int zlo = max(zmin - 1, wz * zdim), zhi = min(zmax + 1, (wz + 1) * zdim - 1);
    if (ok && zlo <= zhi) {
        r.lin = key0 + col_lin * zdim + (zlo - wz * zdim);
        r.b0 = start[r.lin];
        r.cnt = start[r.lin + (zhi - zlo) + 1] - r.b0;
        r.zoff = zlo - zmin;
        r.shp = shp;
        r.code = code << B_BITS;
        r.ox = off[0];
        r.oy = off[1];
    }
    return r;
}

/* the SPH bucket of a DEM particle (as calcFPI searches it) and its FP32 offset there: (offset, bucket key) */
template <int ND>
__device__ __forceinline__ float4 dem_in_sph_grid(const DevCfg &c, const DevState &s, const DevGlobals *g, int64_t i) {
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    int key = 0;
    float o[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const double r = s.row(FD_R + d)[i];
        int kd = c.periodic[d] ? (int)floor((r - c.dmin[d]) * g->rscell[d])
                               : trunc_index(r, c.dmin[d], g->sr2, g->rsr2_f, 3.0);
        kd = kd < 0 ? 0 : (kd >= dims[d] ? dims[d] - 1 : kd);
        key = key * dims[d] + kd;
        o[d] = (float)(r - sph_origin(c, g, d, kd));
    }
    return make_float4(o[0], o[1], o[2], __int_as_float(key));
}

/* Neighbour lists: slot j of particle a, in tiles of 32 particles x 8
 * entries -- each particle's 8 entries contiguous, the 32 particles' groups
 * back to back -- so a warp of consecutive particles reads 8 entries each
 * with two coalesced int4 loads and the build writes a particle's entries in
 * runs.  maxn (the list depth) is a multiple of 8. */
__device__ __forceinline__ int64_t nl_at(int64_t a, int j, int64_t maxn) {
    return ((a >> 5) * maxn + (j & ~7)) * 32 + ((a & 31) << 3) + (j & 7);
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void load_cell32(const DevCfg &c, const DevGlobals *g, float *cell) {
#pragma unroll
    for (int d = 0; d < 3; d++) cell[d] = (float)(c.periodic[d] ? g->scell[d] : g->sr2);
}

/* The 27 stencil shifts o * bucket size, indexed by the list entry's code,
 * in shared memory: one load per pair instead of a decode and three
 * int-to-float conversions.  Every thread of the block must call this. */
__device__ __forceinline__ const float4 *stencil_shifts(const DevCfg &c, const DevGlobals *g) {
    __shared__ float4 tab[27];
    if (threadIdx.x < 27) {
        const int code = threadIdx.x;
        const float o0 = (float)(code / 9 - 1), o1 = (float)((code / 3) % 3 - 1), o2 = (float)(code % 3 - 1);
        float cell[3];
        load_cell32(c, g, cell);
        tab[code] = make_float4(o0 * cell[0], o1 * cell[1], o2 * cell[2], 0.f);
    }
    __syncthreads();
    return tab;
}

template <int ND>
__device__ __forceinline__ void nb_delta_t(int e, const float4 *tab, float4 pa, float4 pb, float *d) {
    const float4 sft = tab[e >> B_BITS];
    d[0] = pa.x - pb.x - sft.x;
    d[1] = ND > 1 ? pa.y - pb.y - sft.y : 0.f;
    d[2] = ND > 2 ? pa.z - pb.z - sft.z : 0.f;
}

__device__ __forceinline__ void block_min_atomic(float v, unsigned long long *target) {
    __shared__ float smin[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) smin[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? smin[lane] : FLT_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0 && v < FLT_MAX) atomic_min_pos(target, (double)v);
    }
}

/* boundary force of sph.h:736-918 in FP32 (b is a repulsive boundary particle) */
template <int ND>
__device__ __noinline__ void boundary32(const DevCfg *__restrict__ cp, const float4 *__restrict__ NB, int b, float d0,
                                        float d1, float d2, float r, float dv0, float dv1, float dv2, float ma, float mb,
                                        float *fbx) {
    const DevCfg &c = *cp;
    const float d[3] = {d0, d1, d2}, dv[3] = {dv0, dv1, dv2};
    const float4 N1 = NB[3 * b], N2 = NB[3 * b + 1], N3 = NB[3 * b + 2];
    const float n1[3] = {N1.x, N1.y, N1.z}, n2[3] = {N2.x, N2.y, N2.z}, nt[3] = {N3.x, N3.y, N3.z};
    float np[3];
    if (n2[0] == 0.f && n2[1] == 0.f && n2[2] == 0.f) {
        for (int k = 0; k < 3; k++) np[k] = n1[k];
    } else {
        const float rd1 = d[0] * n1[0] + d[1] * n1[1] + d[2] * n1[2];
        const float rd2 = d[0] * n2[0] + d[1] * n2[1] + d[2] * n2[2];
        const float rnt = r * r * (n1[0] * n2[0] + n1[1] * n2[1] + n1[2] * n2[2]) - rd1 * rd2;
        if (rnt <= 0.f) {
            for (int k = 0; k < 3; k++) np[k] = d[k] / r;
        } else {
            const float con = N1.w;
            for (int k = 0; k < 3; k++) np[k] = con * (rd1 - rd2) > 0.f ? n1[k] : n2[k];
        }
    }
    const float rperp = np[0] * d[0] + np[1] * d[1] + np[2] * d[2];
    const float rt0 = d[0] - rperp * np[0], rt1 = d[1] - rperp * np[1], rt2 = d[2] - rperp * np[2];
    const float rdelp = c.f_rdelp;
    float pt0, pt1;
    if (ND == 3) {
        pt0 = fabsf(rt0 * nt[0] + rt1 * nt[1] + rt2 * nt[2]);
        const float cx = rt1 * nt[2] - rt2 * nt[1], cy = rt2 * nt[0] - rt0 * nt[2], cz = rt0 * nt[1] - rt1 * nt[0];
        pt1 = sqrtf(cx * cx + cy * cy + cz * cz);
    } else {
        pt0 = sqrtf(rt0 * rt0 + rt1 * rt1);
        pt1 = 0.f;
    }
    const float pd0 = pt0 * rdelp, pd1 = pt1 * rdelp;
    if (!(pd0 <= 1.f && pd1 <= 1.f)) return;
    const float pif = c.f_pi, c0 = c.f_c0;
    const float pesky = 0.25f * (1.f + cosf(pif * pd0)) * (1.f + cosf(pif * pd1));
    const float q = fabsf(rperp) * c.f_rpsep;
    if (!(q < 2.f)) return;
    const int beta = (d[0] * dv[0] + d[1] * dv[1] + d[2] * dv[2]) < 0.f ? 1 : 0;
    const float bigA = 0.01f * c0 * c0 - beta * c0 * (dv[0] * np[0] + dv[1] * np[1] + dv[2] * np[2]);
    const float bfact = 1.f / fabsf(rperp);
    const float QIN = 2.f / 3.f;
    float bforce;
    if (q <= QIN) bforce = bfact * QIN;
    else if (q <= 1.f) bforce = bfact * (2.f * q - 1.5f * q * q);
    else bforce = bfact * 0.5f * (2.f - q) * (2.f - q);
    const float sc = (rperp < 0.f ? -1.f : 1.f) * (2.f * ma / (ma + mb)) * bigA * bforce * pesky;
    for (int k = 0; k < 3; k++) fbx[k] = sc * np[k];
}

/* ---------------------------------------------------------------------- */
/* Neighbour-record staging for the list consumers (TMA bulk copies).
 *
 * A block takes consecutive particles of the bucket order, so most of them
 * lie in one column of buckets along the last axis, and their neighbours in
 * the 3^(d-1) columns around it, over the block's bucket range on the last
 * axis +- one bucket.  Each of those column ranges is a contiguous run of
 * particle slots, so its packed records (P0, P1, P2) are copied global ->
 * shared with one cp.async.bulk per array, completing on one mbarrier.  A
 * list entry's stencil code names its neighbour column, so its record is
 * found in shared memory when its slot lies in that column's staged range,
 * else (another column of the block, a periodic image on the last axis, a
 * range cut at the capacity) read from global memory. */
constexpr int ST_CAP = 1536;    /* staged records per block (2 or 3 x 16 B each) */
constexpr int ST_MAXSLOT = 9;   /* neighbour columns: 3^(d-1) */

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok = 0;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* bounded wait for phase 0 of the staging barrier: false after the limit */
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar) {
    for (int it = 0; it < (1 << 22); it++)
        if (mbar_try_wait(bar, 0)) return true;
    return false;
}

struct Staged {
    const float4 *S0, *S1, *S2;
    const int *lo, *num, *base;
    bool ok;
};

/* the neighbour column of a stencil code (3D: code / 3, 2D: code / 9) */
template <int ND>
__device__ __forceinline__ int st_slot(int code) {
    return ND == 3 ? code / 3 : (ND == 2 ? code / 9 : 0);
}

/* Called by every thread of the block, G threads per particle.  a0: the
 * block's first slot, n_t: the particles in SPH buckets (sorted by bucket key). */
template <int ND, int NARR, int G>
__device__ Staged stage_neighbours(const DevCfg &c, DevGlobals *g, const int *__restrict__ start,
                                   const int *__restrict__ skey, const float4 *__restrict__ P0,
                                   const float4 *__restrict__ P1, const float4 *__restrict__ P2, int64_t a0,
                                   int n_t, float4 *smem) {
    constexpr int Z = ND - 1;
    constexpr int NS = ND == 3 ? 9 : (ND == 2 ? 3 : 1);
    __shared__ int s_lo[ST_MAXSLOT], s_num[ST_MAXSLOT], s_base[ST_MAXSLOT];
    __shared__ int s_col, s_zmin, s_zmax;
    __shared__ __align__(8) unsigned long long s_bar;
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    const int zdim = dims[Z];
    if (threadIdx.x == 0) {
        s_col = skey[a0] / zdim;
        s_zmin = INT_MAX;
        s_zmax = -1;
        mbar_init(&s_bar, 1);
    }
    __syncthreads();
    const int64_t a = a0 + threadIdx.x / G;
    if (a < n_t) {
        const int key = skey[a];
        if (key / zdim == s_col) {
            atomicMin(&s_zmin, key % zdim);
            atomicMax(&s_zmax, key % zdim);
        }
    }
    __syncthreads();
    if (threadIdx.x < NS) {
        const int t = threadIdx.x;
        int o[2] = {0, 0}, cc[2] = {0, 0};
        if (ND == 3) {
            o[0] = t / 3 - 1;
            o[1] = t % 3 - 1;
            cc[0] = s_col / dims[1];
            cc[1] = s_col % dims[1];
        } else if (ND == 2) {
            o[0] = t - 1;
            cc[0] = s_col;
        }
        bool ok = true;
        int col = 0;
#pragma unroll
        for (int d = 0; d < Z; d++) {
            int x = cc[d] + o[d];
            if (x < 0 || x >= dims[d]) {
                ok = ok && c.periodic[d];
                x = x < 0 ? x + dims[d] : x - dims[d];
            }
            col = col * dims[d] + x;
        }
        const int zlo = max(s_zmin - 1, 0), zhi = min(s_zmax + 1, zdim - 1);
        int lo = 0, num = 0;
        if (ok && zlo <= zhi) {
            lo = start[col * zdim + zlo];
            num = start[col * zdim + zhi + 1] - lo;
        }
        s_lo[t] = lo;
        s_num[t] = num;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int base = 0;
        for (int t = 0; t < NS; t++) {
            const int num = min(s_num[t], ST_CAP - base);
            s_num[t] = num;
            s_base[t] = base;
            base += num;
        }
        mbar_expect_tx(&s_bar, (unsigned)(NARR * 16 * base));
        for (int t = 0; t < NS; t++) {
            const int num = s_num[t];
            if (num <= 0) continue;
            const unsigned bytes = (unsigned)(16 * num);
            bulk_g2s(smem + s_base[t], P0 + s_lo[t], bytes, &s_bar);
            bulk_g2s(smem + ST_CAP + s_base[t], P1 + s_lo[t], bytes, &s_bar);
            if (NARR > 2) bulk_g2s(smem + 2 * ST_CAP + s_base[t], P2 + s_lo[t], bytes, &s_bar);
        }
    }
    __syncthreads();
    Staged st;
    st.S0 = smem;
    st.S1 = smem + ST_CAP;
    st.S2 = smem + 2 * ST_CAP;
    st.lo = s_lo;
    st.num = s_num;
    st.base = s_base;
    bool ok = mbar_wait_bounded(&s_bar);
    if (!ok) {
        /* gave up: record it, and keep the block alive (again bounded) until
         * the copies into its shared memory have landed */
        set_err(g, SPHDEM_ERR_TIMEOUT, 1);
        mbar_wait_bounded(&s_bar);
    }
    /* the whole block gives up together */
    st.ok = !__syncthreads_or(!ok);
    return st;
}

}  // namespace
}  // namespace sphdem

#define SPHDEM_ND_DISPATCH(nd, F) \
    do {                          \
        if ((nd) == 3) {          \
            F(3);                 \
        } else if ((nd) == 2) {   \
            F(2);                 \
        } else {                  \
            F(1);                 \
        }                         \
    } while (0)
