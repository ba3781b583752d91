/*
 * Mixed-precision pair passes (SPHDEM_PREC_MIXED).
 *
 * Positions stay FP64 in the state; for the pair math every particle is
 * packed, once per rebuild, as an FP32 offset from the FP64 origin of its own
 * bucket plus FP32 h / velocity / mass / density / pdr2.  The displacement of
 * a pair in buckets ca and cb = ca + o is (off_a - off_b) - o*bucket, all FP32
 * and well conditioned (|off| < one bucket).  Every kernel is specialised on
 * the dimension so per-axis arrays live in registers.
 *
 *   k_nlist      after each rebuild, the exact neighbour list of every
 *                sph/sphBoundary particle: candidates of the 3^d stencil in
 *                FP32 with a proven error bound; those inside the bound are
 *                settled by the reference's FP64 predicate (particle.h:236-238).
 *                Periodic
 *                images only where the reference holds a ghost.  Entries
 *                b | stencil code << 26 in tiles of 32 particles x 8 slots
 *                (nl_at).
 *   k_eos32      the FP64 EOS (its (rho/rho0)^7-1 cancels too much for FP32)
 *   k_force      calcForce + the Courant/viscous/accel dt conditions, any form
 *   k_dddt       calcDddtDudt, with CORRECTED_GRADIENT and in 1D
 * The force and continuity passes of the usual forms are in lists32.cu, the
 * SPH-DEM coupling and contact passes in coupling.cu.
 *
 * Sums are Kahan-compensated in FP32 and added to the FP64 state once per
 * particle.  Roofline: the list passes are FP32-pipe-bound on 3D workloads
 * (~80 FP32 FLOP per listed pair against 4 B of list + 48 B of packed input).
 */
#include <algorithm>
#include <type_traits>
#include <vector>

#include "mixed.cuh"

namespace sphdem {
namespace {

/* ---------------------------------------------------------------------- */
/* P0 = (offset from own bucket origin, h), P1 = (vhat, mass; negated for
 * particles that are neither sph / sphBoundary nor DEM), P2 = (dens, pdr2, cF,
 * 1/h) for the middle phase and (dens, cF, porosity, 1/h) for the end phase,
 * where cF = -10 C / h^(d+2) is the factor of the Wendland gradient F(r, h) =
 * cF (2 - r/h)^3, tg = type | gcode << 8.  cF follows from the FP32 1/h next to
 * it, so that factor and argument belong to one kernel: with cF of the FP64 h the
 * rounding of 1/h stays in (2 - r/h)^3 alone, an error of one sign in a run with
 * constant h (of the pairs' moment sum F r^2, rms over h: 1.3e-7 in 3D, in this
 * form 2.9e-8) */
template <int ND>
__global__ void k_pack(DevCfg c, DevState s, const int *__restrict__ skey, const DevGlobals *__restrict__ g,
                       float4 *__restrict__ P0, float4 *__restrict__ P1, float4 *__restrict__ P2,
                       int *__restrict__ tg, int middle, float4 *__restrict__ DS, float4 *__restrict__ NB, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = s.irow(FI_IAM)[i];
    tg[i] = (t & 0xff) | (s.irow(FI_GCODE)[i] << 8);
    if (t == T_DEAD) return;
    const int key = skey[i];
    float off[3] = {0.f, 0.f, 0.f};
    int cc[3] = {0, 0, 0};
    const bool dem = c.liq_dem() && t == T_DEM;
    if (dem) {
        decode<ND>(key - g->n_sph_cells, c.ddims, cc);
    } else {
        const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
        decode<ND>(key, dims, cc);
    }
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const double o = s.row(FD_R + d)[i] - (dem ? dem_origin(c, d, cc[d]) : sph_origin(c, g, d, cc[d]));
        off[d] = (float)o;
    }
    float vh[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < ND; d++) vh[d] = (float)s.row(FD_VHAT + d)[i];
    P0[i] = make_float4(off[0], off[1], off[2], (float)s.row(FD_H)[i]);
    /* the mass of a particle that is neither sph / sphBoundary nor DEM is
     * stored negated: list readers take a neighbour's type from the sign and
     * load the type row only for those (walls) */
    const float mpk = (float)s.row(FD_MASS)[i];
    P1[i] = make_float4(vh[0], vh[1], vh[2], (is_sph_or_sphb(t) || dem) ? mpk : -mpk);
    const float ih = (float)s.row(FD_IH)[i];
    const float cF = scaled_power<ND + 2>(ih, c.f_grad[0], c.f_grad[1]);
    P2[i] = make_float4((float)s.row(FD_DENS)[i], middle ? (float)s.row(FD_PDR2)[i] : cF,
                        middle ? cF : (float)s.row(FD_POR)[i], ih);
    if (is_boundary(t)) {
        float nv[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll
        for (int k = 0; k < ND; k++) {
            nv[0][k] = (float)s.row(FD_N1 + k)[i];
            nv[1][k] = (float)s.row(FD_N2 + k)[i];
            nv[2][k] = ND == 3 ? (float)s.row(FD_N3 + k)[i] : 0.f;
        }
        NB[3 * i] = make_float4(nv[0][0], nv[0][1], nv[0][2], s.irow(FI_CONCAVE)[i] ? 1.f : -1.f);
        NB[3 * i + 1] = make_float4(nv[1][0], nv[1][1], nv[1][2], 0.f);
        NB[3 * i + 2] = make_float4(nv[2][0], nv[2][1], nv[2][2], 0.f);
    }
    if (dem && middle) s.row(FD_SHEP)[i] = 0.0; /* the porosity pass adds into it */
    if (dem && !middle) DS[i] = dem_in_sph_grid<ND>(c, s, g, i);
}

/* ---------------------------------------------------------------------- */
/* Neighbour-list build.
 *
 * A warp takes 32 consecutive particles of the bucket order.  Buckets are
 * numbered with the last axis fastest, so those particles lie in one or two
 * runs of consecutive buckets along that axis (a "column").  For each run
 * the warp stages the candidates of the union of the runs' 3^d stencils --
 * 3^(d-1) neighbour columns x the run's z-range +-1 -- in shared memory,
 * with positions moved into the run's frame (coalesced loads; the periodic
 * image filter and the distance to the run's bounding box are applied once
 * per candidate), then every lane tests all staged candidates with broadcast
 * shared-memory reads.  Sharing the stencil across a run keeps all 32 lanes
 * busy whatever the bucket occupancy.
 *
 * A passing candidate is appended by its lane to the lane's column of a
 * shared-memory queue (slot-major, so the stores never conflict) with one
 * predicated store and add, without a branch; when a lane's column is half
 * full, every lane moves its complete groups of 8 entries to its list tile, a
 * whole sector per group.  The pass is bound by instruction issue, so two
 * candidates share each FP32 operation (packed f32x2: 10 instructions a
 * candidate and warp instead of 13), the append is part of the test loop, and
 * candidates are cut to those within reach of the run's bounding box (23 %
 * fewer on a 3D lattice).
 *
 * FP32 error bound of the test (L = largest offset magnitude in the frame,
 * R = 2 max(ha, hb)): each displacement component carries < 6 * 2^-24 L, so
 * r^2 is off by < 1.25e-6 L max(L, R) + 1.8e-7 r^2 and the cut-off
 * 4 max(ha^2, hb^2) by < 1.8e-7 of itself.  A candidate passes up to
 * 4 h^2 (1 + 5e-7) + 1.5e-6 L^2; one that passes by less than the width of
 * the band of doubt is settled on the spot (settle_band), which also takes
 * the particle itself out, so the lists hold exactly the neighbours.  The
 * lane only keeps the smallest margin of 32 candidates; the rare 32 with a
 * doubtful one (or the particle itself) are gone over again.
 * Bound by instruction issue, and from a lattice at rest (eight exact ties a
 * particle) by the chains of the FP64 decisions: the two builds of a coupled step of 1.08 M
 * particles take 1.25 ms; tests into a bit mask, entries then spread over the
 * warp and a second kernel for the candidates in doubt took 2.68. */
constexpr int NL_WARPS = 4;
constexpr int NL_CAP = 128;   /* staged candidates per warp before they are tested */
constexpr int NL_QN = 64;     /* queue slots per lane: moved on when over 32 are taken, 32 come at most per round */
/* buckets of a run, less one: the staged set of a run grows with its length
 * along the last axis, that of a run cut short with its two ends; in 2D a
 * bucket holds ~7 particles, so 32 of them span five */
template <int ND>
constexpr int NL_RUN = ND == 3 ? 2 : (ND == 2 ? 6 : 14);

/* A candidate whose FP32 test leaves doubt: list entry e (candidate and stencil
 * code) of particle a in bucket cc, zd its bucket on the last axis relative to
 * a's.  Buckets are at least 2h wide, so one outside a's own 3^d stencil is no
 * neighbour; for all others the reference's FP64 predicate decides.  (A
 * double-float refinement before it settled nothing for the exact ties of
 * particles at rest on a lattice, which are nearly all of these candidates,
 * and doubled the latency of their chain.) */
template <int ND>
__device__ __forceinline__ bool settle_band(const DevCfg *__restrict__ cp, const DevState &s, const int *dims, const int *cc,
                                            int a, int e, int zd) {
    if (zd < -1 || zd > 1) return false;
    int o[3], sh[3] = {0, 0, 0};
    nl_decode_code(e >> B_BITS, o);
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const int t = cc[d] + o[d];
        sh[d] = t < 0 ? -1 : (t >= dims[d] ? 1 : 0);
    }
    return exact_pair<ND>(cp, s, a, e & B_MASK, sh[0], sh[1], sh[2], 0.0, 0);
}

/* append e to the lane's queue column (next free slot at shared address qa) when margin >= 0, without a branch */
__device__ __forceinline__ void queue_append(unsigned &qa, int e, float margin) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ge.f32 p, %2, 0f00000000;\n @p st.shared.u32 [%0], %1;\n @p add.u32 %0, %0, 128;\n}\n"
        : "+r"(qa)
        : "r"(e), "f"(margin)
        : "memory");
}

/* G lanes per particle: a warp takes 32 / G consecutive particles and each of
 * a particle's lanes tests every G-th group of four candidates.  G = 1 reads
 * the fewest candidates per particle; G = 4 runs four times the warps, each a
 * third as long, for populations that leave the chip short of warps. */
template <int ND, bool COUNT, int G>
__global__ void __launch_bounds__(NL_WARPS * 32, 5) k_nlist(DevCfg c, const DevCfg *__restrict__ cp, DevState s,
                                                         const int *__restrict__ start, const int *__restrict__ skey,
                                                         DevGlobals *__restrict__ g, const float4 *__restrict__ P0,
                                                         const int *__restrict__ tg, int *__restrict__ nbr,
                                                         int *__restrict__ ncnt, int maxn, int soft,
                                                         int *__restrict__ bandn) {
    constexpr int Z = ND - 1;
    constexpr unsigned FULL = 0xffffffffu;
    /* staged candidates: negated position in the run's frame, cut-off, list
     * entry (its code counts buckets on the last axis from the run's first) */
    __shared__ __align__(16) float s_x[NL_WARPS][3][NL_CAP], s_cut[NL_WARPS][NL_CAP];
    __shared__ __align__(16) int s_ent[NL_WARPS][NL_CAP];
    __shared__ int s_queue[NL_WARPS][NL_QN * 32];
    __shared__ unsigned char s_zr[NL_WARPS][NL_CAP];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    float(*cx)[NL_CAP] = s_x[w];
    float *ccut = s_cut[w];
    int *cent = s_ent[w];
    unsigned char *czr = s_zr[w];
    int *const queue = s_queue[w] + lane;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int nsc = g->n_sph_cells;
    const int n_t = start[nsc];
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    const int zdim = dims[Z];
    float cell[3];
    float l_other = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        cell[d] = (float)(c.periodic[d] ? g->scell[d] : g->sr2);
        if (d < Z) l_other = fmaxf(l_other, 2.f * cell[d]);
    }
    const float cz = cell[Z];
    /* code of the run's own column, one bucket below its first */
    int code_own = 0;
#pragma unroll
    for (int d = 0; d < 3; d++)
        if (d != Z) code_own += code_stride(d);
    const int zstride = code_stride(Z) << B_BITS;
    const float supp = (float)(2.0 * g->sr) * (1.f + 1e-5f) + 1e-5f * cz;
    const float K_HI = 4.f * (1.f + 5e-7f);

    constexpr int PP = 32 / G; /* particles per warp */
    const int sub = lane % G;
    for (int t0 = (blockIdx.x * NL_WARPS + w) * PP; t0 < n_t; t0 += NL_WARPS * gridDim.x * PP) {
        const int a = t0 + lane / G;
        /* the warp's particles share one column of list tiles: entry j of
         * particle a sits at tiles + (j & ~7) * 32 + (j & 7) */
        int4 *const tiles = reinterpret_cast<int4 *>(nbr + (int64_t)(a >> 5) * maxn * 32 + (a & 31) * 8);
        bool act = false;
        int key = 0;
        if (a < n_t) {
            key = skey[a];
            act = is_sph_or_sphb(tg[a] & 0xff);
        }
        int cc[3] = {0, 0, 0};
        decode<ND>(key, dims, cc);
        const int col = key / zdim;
        float4 pa0 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (act) pa0 = P0[a];
        /* entries in the list tiles (a multiple of 8) and waiting in the queue;
         * band candidates; what turns a staged entry's code into this lane's */
        int cnt = 0, qn = 0, nb = 0, adj = 0;
        /* complete groups of 8 go to the tile, the rest to the queue's front; with
         * several lanes per particle, all entries, one lane's after the other's */
        auto flush = [&]() {
            if (G > 1) {
                int off = qn;
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    const int v = __shfl_up_sync(FULL, off, o, G);
                    if (sub >= o) off += v;
                }
                const int all = __shfl_sync(FULL, off, G - 1, G);
                off += cnt - qn;
                int *const e = reinterpret_cast<int *>(tiles);
                for (int k = 0; k < qn; k++)
                    if (off + k < maxn) e[((off + k) & ~7) * 32 + ((off + k) & 7)] = queue[k << 5] + adj;
                cnt += all;
                qn = 0;
                return;
            }
            int h = 0;
            for (; __any_sync(FULL, qn - h >= 8); h += 8) {
                if (qn - h < 8) continue;
                if (cnt + 8 <= maxn) {
                    const int *q = queue + (h << 5);
                    tiles[cnt * 8] = make_int4(q[0] + adj, q[32] + adj, q[64] + adj, q[96] + adj);
                    tiles[cnt * 8 + 1] = make_int4(q[128] + adj, q[160] + adj, q[192] + adj, q[224] + adj);
                }
                cnt += 8;
            }
            const int done = qn & ~7;
            qn &= 7;
            if (done)
                for (int k = 0; k < qn; k++) queue[k << 5] = queue[(done + k) << 5];
        };
        unsigned pending = __ballot_sync(FULL, act);
        while (pending) {
            /* a run: lanes in the leader's column within a few buckets of it */
            const int leader = __ffs(pending) - 1;
            const int lcol = __shfl_sync(FULL, col, leader);
            const int zmin = __shfl_sync(FULL, cc[Z], leader);
            const unsigned gmask = __ballot_sync(FULL, act && col == lcol && cc[Z] <= zmin + NL_RUN<ND>) & pending;
            pending &= ~gmask;
            const int zmax = __shfl_sync(FULL, cc[Z], 31 - __clz(gmask));
            int ccol[3] = {0, 0, 0};
#pragma unroll
            for (int d = 0; d < Z; d++) ccol[d] = __shfl_sync(FULL, cc[d], leader);
            const bool mine = (gmask >> lane) & 1u;
            /* this lane's particle in the run's frame; others sit far away */
            float pv[3] = {1e30f, 1e30f, 1e30f};
            const int my_zr = cc[Z] - zmin + 1;
            float thr_a = -1.f;
            const float L = fmaxf(l_other, (float)(zmax - zmin + 2) * cz);
            const float EPS = 1.5e-6f * L * L;
            if (mine) {
                pv[0] = pa0.x;
                pv[1] = pa0.y;
                pv[2] = pa0.z;
                pv[Z] += (float)(my_zr - 1) * cz;
                adj = (int)((unsigned)(1 - my_zr) * (unsigned)zstride);
                thr_a = fmaf(pa0.w * pa0.w, K_HI, EPS);
            }
            /* width of the band of doubt below the FP32 cut-off: 1e-6 (2h)^2 + 3 EPS */
            const float W = 1.01f * (1e-6f * supp * supp + 3.f * EPS);
            /* the run's bounding box: a candidate further from it than the largest
             * support 2 sr >= 2 max(h), plus a rounding margin, is no neighbour */
            float blo[3], bhi[3];
#pragma unroll
            for (int d = 0; d < ND; d++) {
                blo[d] = pv[d];
                bhi[d] = mine ? pv[d] : -1e30f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    blo[d] = fminf(blo[d], __shfl_xor_sync(FULL, blo[d], o));
                    bhi[d] = fmaxf(bhi[d], __shfl_xor_sync(FULL, bhi[d], o));
                }
            }
            /* the run's own particles are the first candidates; each lane skips its own */
            const int self_j = __popc(gmask & lt_mask) / G;
            int nst = __popc(gmask) / G;
            if (mine && sub == 0) {
#pragma unroll
                for (int d = 0; d < ND; d++) cx[d][self_j] = -pv[d];
                ccut[self_j] = thr_a;
                cent[self_j] = (int)((unsigned)(a | (code_own << B_BITS)) + (unsigned)my_zr * (unsigned)zstride);
                czr[self_j] = (unsigned char)my_zr;
            }
            /* the four staged candidates from j on */
            struct Four {
                float4 x, y, z, cut;
                int4 e;
            };
            auto load4 = [&](int j) {
                Four f;
                f.x = *reinterpret_cast<const float4 *>(cx[0] + j);
                if (ND > 1) f.y = *reinterpret_cast<const float4 *>(cx[1] + j);
                if (ND > 2) f.z = *reinterpret_cast<const float4 *>(cx[2] + j);
                f.cut = *reinterpret_cast<const float4 *>(ccut + j);
                f.e = *reinterpret_cast<const int4 *>(cent + j);
                return f;
            };
            /* test 32 staged candidates; SELF: the lane's own particle may be among
             * them.  The next four are loaded before the current four are appended,
             * as a load cannot pass the appends' stores.  Returns the smallest margin. */
            auto round32 = [&](auto self_tag, int j0) {
                constexpr bool SELF = decltype(self_tag)::value;
                const unsigned qbase = smem_u32(queue);
                unsigned qa = qbase + (qn << 7);
                unsigned near = 0xffffffffu;
                const float2 ax = make_float2(pv[0], pv[0]), ay = make_float2(pv[1], pv[1]), az = make_float2(pv[2], pv[2]);
                Four f = load4(j0 + 4 * sub);
#pragma unroll
                for (int jb = 0; jb < 32; jb += 4 * G) {
                    const int jj = jb + 4 * sub;
                    Four nx = f;
                    if (jb + 4 * G < 32) nx = load4(j0 + jj + 4 * G);
                    float2 d = __fadd2_rn(ax, make_float2(f.x.x, f.x.y)), e = __fadd2_rn(ax, make_float2(f.x.z, f.x.w));
                    float2 r = __fmul2_rn(d, d), q = __fmul2_rn(e, e);
                    if (ND > 1) {
                        d = __fadd2_rn(ay, make_float2(f.y.x, f.y.y));
                        e = __fadd2_rn(ay, make_float2(f.y.z, f.y.w));
                        r = __ffma2_rn(d, d, r);
                        q = __ffma2_rn(e, e, q);
                    }
                    if (ND > 2) {
                        d = __fadd2_rn(az, make_float2(f.z.x, f.z.y));
                        e = __fadd2_rn(az, make_float2(f.z.z, f.z.w));
                        r = __ffma2_rn(d, d, r);
                        q = __ffma2_rn(e, e, q);
                    }
                    const float df[4] = {fmaxf(thr_a, f.cut.x) - r.x, fmaxf(thr_a, f.cut.y) - r.y,
                                         fmaxf(thr_a, f.cut.z) - q.x, fmaxf(thr_a, f.cut.w) - q.y};
                    const int ev[4] = {f.e.x, f.e.y, f.e.z, f.e.w};
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (COUNT) {
                            qn += df[u] >= 0.f;
                            continue;
                        }
                        near = min(near, __float_as_uint(df[u])); /* negative: above every width */
                        queue_append(qa, ev[u], SELF && j0 + jj + u == self_j ? -1.f : df[u]);
                    }
                    f = nx;
                }
                if (!COUNT) qn = (int)(qa - qbase) >> 7;
                return near;
            };

            /* Range table, one lane per (neighbour column, period piece): the
             * column's buckets zmin-1 .. zmax+1 cut at the periodic seam into at
             * most 3 runs of consecutive keys.  All lanes load their bucket range
             * at once; the ranges are then gathered one after the other, 64
             * candidates at a time, and tested when 64 and more are staged. */
            const RangeEntry re = range_entry<ND>(lane, ccol, zmin, zmax, dims, c.periodic, cell, 0, start);
            unsigned live = __ballot_sync(FULL, re.cnt > 0);
            int b0 = 0, num = 0, lin = 0, zoff = 0, code = 0, shp = 0x15, t = 0;
            float ox = 0.f, oy = 0.f;
            bool first = true;
            for (bool last = false; !last;) {
                while (nst <= NL_CAP - 64) {
                    if (t >= num) {
                        last = live == 0;
                        if (last) break;
                        const int src = __ffs(live) - 1;
                        live &= live - 1;
                        b0 = __shfl_sync(FULL, re.b0, src);
                        num = __shfl_sync(FULL, re.cnt, src);
                        lin = __shfl_sync(FULL, re.lin, src);
                        zoff = __shfl_sync(FULL, re.zoff, src);
                        code = __shfl_sync(FULL, re.code, src);
                        shp = __shfl_sync(FULL, re.shp, src);
                        ox = __shfl_sync(FULL, re.ox, src);
                        oy = __shfl_sync(FULL, re.oy, src);
                        t = 0;
                    }
                    const int shv[3] = {(shp & 3) - 1, ((shp >> 2) & 3) - 1, ((shp >> 4) & 3) - 1};
                    float4 pb[2];
                    int kb[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int k = b0 + min(t + lane + 32 * u, num - 1);
                        pb[u] = P0[k];
                        kb[u] = skey[k];
                    }
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int k = b0 + t + lane + 32 * u;
                        bool valid = t + lane + 32 * u < num;
                        const int zrel = zoff + (kb[u] - lin);
                        float qv[3] = {pb[u].x, pb[u].y, pb[u].z};
                        if (Z > 0) qv[0] += ox;
                        if (Z > 1) qv[1] += oy;
                        qv[Z] += (float)zrel * cz;
                        float far2 = 0.f;
#pragma unroll
                        for (int d = 0; d < ND; d++) {
                            const float f = fmaxf(0.f, fmaxf(blo[d] - qv[d], qv[d] - bhi[d]));
                            far2 = fmaf(f, f, far2);
                        }
                        valid = valid && far2 <= supp * supp;
                        if (shp == 0x15)
                            valid = valid && !((unsigned)(k - t0) < (unsigned)PP && ((gmask >> ((k - t0) * G)) & 1u));
                        else if (valid)
                            valid = img_ok<ND>(tg[k] >> 8, shv);
                        const unsigned m = __ballot_sync(FULL, valid);
                        if (valid) {
                            const int pos = nst + __popc(m & lt_mask);
#pragma unroll
                            for (int d = 0; d < ND; d++) cx[d][pos] = -qv[d];
                            ccut[pos] = fmaf(pb[u].w * pb[u].w, K_HI, EPS);
                            /* k | code of the candidate's bucket relative to the run's
                             * first bucket - 1; adj adds the lane's own offset */
                            cent[pos] = (int)((unsigned)(k | code) + (unsigned)(zrel + 1) * (unsigned)zstride);
                            czr[pos] = (unsigned char)(zrel + 1);
                        }
                        nst += __popc(m);
                    }
                    t += 64;
                }
                /* test the complete rounds of 32 and keep the rest, or (last) all of
                 * them, padded with far-away candidates */
                if (last && lane < ((32 - (nst & 31)) & 31)) {
#pragma unroll
                    for (int d = 0; d < ND; d++) cx[d][nst + lane] = 1e30f;
                    ccut[nst + lane] = -1.f;
                }
                __syncwarp();
                const int end = last ? (nst + 31) & ~31 : nst & ~31;
#pragma unroll 1
                for (int j0 = 0; j0 < end; j0 += 32) {
                    const int q0 = qn;
                    const unsigned near = first ? round32(std::true_type{}, j0) : round32(std::false_type{}, j0);
                    const bool own_round = first;
                    first = false;
                    if (COUNT) continue;
                    __syncwarp();
                    const bool doubt = near <= __float_as_uint(W);
                    if (__any_sync(FULL, doubt)) {
                        /* some candidate within the band of doubt: the round's pass mask
                         * again, its doubtful bits settled, all lanes one of theirs at a
                         * time (walls at rest have a score of exact ties each), and the
                         * entries written anew */
                        unsigned pass = 0u, open = 0u;
                        if (doubt) {
#pragma unroll 4
                            for (int jj = 0; jj < 32; jj++) {
                                if (G > 1 && ((jj >> 2) % G) != sub) continue;
                                const int j = j0 + jj;
                                const float dx = pv[0] + cx[0][j], dy = ND > 1 ? pv[1] + cx[1][j] : 0.f;
                                const float dz = ND > 2 ? pv[2] + cx[2][j] : 0.f;
                                const float df = fmaxf(thr_a, ccut[j]) - fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                                if (df >= 0.f) pass |= 1u << jj;
                                if (df >= 0.f && df <= W) open |= 1u << jj;
                            }
                            if (own_round) {
                                pass &= ~(1u << self_j);
                                open &= pass;
                            }
                            nb += __popc(open);
                        }
                        while (__any_sync(FULL, open)) {
                            if (open) {
                                const int jj = __ffs(open) - 1, j = j0 + jj;
                                open &= open - 1;
                                if (!settle_band<ND>(cp, s, dims, cc, a, cent[j] + adj, (int)czr[j] - my_zr))
                                    pass &= ~(1u << jj);
                            }
                            __syncwarp();
                        }
                        if (doubt) {
                            qn = q0;
                            for (; pass; pass &= pass - 1) {
                                queue[qn << 5] = cent[j0 + __ffs(pass) - 1];
                                qn++;
                            }
                        }
                        __syncwarp();
                    }
                    if (__any_sync(FULL, qn > NL_QN - 32)) flush();
                }
                if (last) break;
                nst -= end;
                float x[3] = {0.f, 0.f, 0.f}, cut = 0.f;
                int e = 0;
                unsigned char zr = 0;
                if (lane < nst) {
#pragma unroll
                    for (int d = 0; d < ND; d++) x[d] = cx[d][end + lane];
                    cut = ccut[end + lane];
                    e = cent[end + lane];
                    zr = czr[end + lane];
                }
                __syncwarp();
                if (lane < nst) {
#pragma unroll
                    for (int d = 0; d < ND; d++) cx[d][lane] = x[d];
                    ccut[lane] = cut;
                    cent[lane] = e;
                    czr[lane] = zr;
                }
            }
            __syncwarp();
        }
        if (COUNT) {
            if (act) ncnt[a] = qn;
            continue;
        }
        flush();
        if (G > 1) {
#pragma unroll
            for (int o = 1; o < G; o <<= 1) nb += __shfl_xor_sync(FULL, nb, o);
            if (sub) continue;
        }
        if (act) {
            /* the last, incomplete group */
            if (G == 1 && qn > 0 && cnt + 8 <= maxn) {
                int v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) v[k] = k < qn ? queue[k << 5] + adj : -1;
                tiles[cnt * 8] = make_int4(v[0], v[1], v[2], v[3]);
                tiles[cnt * 8 + 1] = make_int4(v[4], v[5], v[6], v[7]);
            }
            cnt += qn;
            /* stored counts never exceed the list depth; an overflow is an error, or
             * (soft) marked for the reader, which then scans the buckets */
            ncnt[a] = cnt <= maxn ? cnt : (soft ? -1 : maxn);
            if (cnt > maxn && !soft) set_err(g, SPHDEM_ERR_CAPACITY, cnt);
        }
        if (a < n_t) bandn[a] = nb;
    }
}

/* ---------------------------------------------------------------------- */
__global__ void __launch_bounds__(BLK) k_eos32(DevCfg c, DevState s, float4 *__restrict__ P2, const int *__restrict__ tg,
                                              int64_t n) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(tg[a] & 0xff)) return;
    /* FP64: p = PRB((rho/rho0)^7 - 1) cancels; one FP64 reciprocal by
     * an FP32 estimate and a Newton step, integer powers */
    const double densa = s.row(FD_DENS)[a];
    const double rho0 = c.liq_dem() ? c.refd * s.row(FD_POR)[a] : c.refd;
    double r0 = (double)(1.0f / (float)rho0);
    r0 = r0 * (2.0 - rho0 * r0);
    const double x = densa * r0;
    double xg;
    if (!c.liq_dem() || c.gamma == 7.0) {
        const double x2 = x * x;
        xg = x2 * x2 * x2 * x;
    } else {
        xg = pow(x, c.gamma);
    }
    double rd = (double)(1.0f / (float)densa);
    rd = rd * (2.0 - densa * rd);
    const double press = c.prb * (xg - 1.0);
    const double pdr2 = press * (rd * rd);
    s.row(FD_PRESS)[a] = press;
    s.row(FD_PDR2)[a] = pdr2;
    P2[a].y = (float)pdr2;
}

/* ---------------------------------------------------------------------- */
/* The general force and continuity passes: every physics class that
 * lists32.cu has no specialised pass for (1D, Monaghan viscosity,
 * anticlumping, CORRECTED_GRADIENT), read from the configuration. */
enum : int { PHYS_GENERIC = 0, PHYS_CG = 3 };

/* CORRECTED_GRADIENT in FP32 (sph.h:325-326): the corrected gradient of a
 * pair is invM_a ((dr F - sumGrad_a/sum_a) / sum_a); invM_a, sumGrad_a and
 * sum_a come from calcInvM (FP64, k_invm) once per rebuild and enter each
 * owner's pair loop as M = invM_a / sum_a and cs = sumGrad_a / sum_a. */
template <int ND>
struct Cg32 {
    float m[ND * ND], cs[ND];
    __device__ __forceinline__ void load(const double *cg, int64_t cap, int64_t a) {
        const double sum = cg[CG_S * cap + a];
#pragma unroll
        for (int k = 0; k < ND * ND; k++) m[k] = (float)(cg[(CG_M + k) * cap + a] / sum);
#pragma unroll
        for (int d = 0; d < ND; d++) cs[d] = (float)cg[(CG_C + d) * cap + a];
    }
    /* out = M (d F - cs) */
    __device__ __forceinline__ void apply(const float *d, float F, float *out) const {
        float t[ND];
#pragma unroll
        for (int k = 0; k < ND; k++) t[k] = d[k] * F - cs[k];
#pragma unroll
        for (int i = 0; i < ND; i++) {
            float v = 0.f;
#pragma unroll
            for (int j = 0; j < ND; j++) v = fmaf(m[i * ND + j], t[j], v);
            out[i] = v;
        }
    }
};

template <int ND, int PHYS, bool TILE>
__global__ void __launch_bounds__(BLK) k_force(DevCfg c, const DevCfg *__restrict__ cp, DevState s, DevGlobals *__restrict__ g,
                                               const float4 *__restrict__ P0, const float4 *__restrict__ P1,
                                               const float4 *__restrict__ P2,
                                               const int *__restrict__ tg, const int *__restrict__ nbr,
                                               const int *__restrict__ ncnt, int64_t ld, int64_t n,
                                               const float4 *__restrict__ NB, const double *__restrict__ cgrows,
                                               const int *__restrict__ start, const int *__restrict__ skey) {
    constexpr bool CG = PHYS == PHYS_CG;
    const float4 *shift = stencil_shifts(c, g);
    extern __shared__ float4 st_smem[];
    Staged st = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, false};
    if constexpr (TILE) {
        const int n_t = start[g->n_sph_cells];
        const int64_t a0 = blockIdx.x * (int64_t)blockDim.x;
        if (a0 >= n_t) return;  /* no list owner in this block */
        st = stage_neighbours<ND, 3, 1>(c, g, start, skey, P0, P1, P2, a0, n_t, st_smem);
        if (!st.ok) return;
    }
    const int visc = c.visc;
    const bool var_h = c.var_h();
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    float ndt = FLT_MAX;
    const int ta = a < n ? (tg[a] & 0xff) : -1;
    if (is_sph_or_sphb(ta)) {
        const float wcon = (float)c.wcon;
        const float4 pa = P0[a], va = P1[a], xa = P2[a];
        const float ha = pa.w, iha = xa.w;
        const float ihn2a = powi<ND>(iha) * iha * iha;
        const float densa = xa.x, pdr2a = xa.y, ma = va.w;
        /* VAR_H_CORRECTION: every gradient of a's sums carries 1/Omega_a
         * (gA = ga/Omega_a, gB = gb/Omega_a), so Omega_a (calcOmega,
         * sph.h:438-451) is summed in this same loop and the gradient sums
         * are scaled once at the end */
        const float ihna = powi<ND>(iha), pd_coef = ND * ihna * iha;
        Plain om;
        om.init(-ma * pd_coef * wK32(0.f, wcon));
        const bool sph = ta == T_SPH;
        const bool anti = !(c.flags & SPHDEM_F_NO_ANTICLUMPING);
        const float visc_nu = (float)c.viscosity, c0 = (float)c.spsound;
        const float liq_visc = (float)(2.0 * c.viscosity * c.dens);
        const float alpha_mon = (float)c.alpha_mon, alpha_art = (float)c.alpha_art;
        const float vdc = visc == SPHDEM_VISC_MONAGHAN ? 0.06f : 0.125f;
        const float k_anti_inv = c.k_anti != 0 ? (float)(1.0 / c.k_anti) : 0.f;
        Cg32<ND> cgw;
        if constexpr (CG) cgw.load(cgrows, s.cap, a);
        Kahan fp[ND], fv[ND], fb[ND], fa[ND];
        Kahan fq;  /* anticlumping: the same term on every component, not scaled by 1/Omega */
        fq.init(0.f);
#pragma unroll
        for (int k = 0; k < ND; k++) {
            fp[k].init(0.f);
            fv[k].init(0.f);
            fb[k].init(0.f);
            fa[k].init(0.f);
        }
        float hmin = FLT_MAX; /* smallest hav of the fluid pairs */
        const int cnt = ncnt[a];
        /* 8 entries at a time from the particle's list tiles (two int4 loads) */
        const int4 *tile = reinterpret_cast<const int4 *>(nbr + nl_at(a, 0, ld));
        int4 q0 = make_int4(-1, -1, -1, -1), q1 = q0;
#pragma unroll 2
        for (int j = 0; j < cnt; j++) {
            if ((j & 7) == 0) {
                q0 = __ldg(tile + (j >> 3) * 64);
                q1 = __ldg(tile + (j >> 3) * 64 + 1);
            }
            const int e = q0.x;
            q0 = make_int4(q0.y, q0.z, q0.w, q1.x);
            q1 = make_int4(q1.y, q1.z, q1.w, -1);
            if (e < 0) continue;
            const int b = e & B_MASK;
            float4 pb, vb, xb;
            if constexpr (TILE) {
                const int sl = st_slot<ND>(e >> B_BITS);
                const int off = b - st.lo[sl];
                if ((unsigned)off < (unsigned)st.num[sl]) {
                    const int k = st.base[sl] + off;
                    pb = st.S0[k];
                    vb = st.S1[k];
                    xb = st.S2[k];
                } else {
                    pb = P0[b];
                    vb = P1[b];
                    xb = P2[b];
                }
            } else {
                pb = P0[b];
                vb = P1[b];
                xb = P2[b];
            }
            /* sph / sphBoundary unless the packed mass is negative */
            const int tb = vb.w < 0.f ? (tg[b] & 0xff) : T_SPH;
            float d[3];
            nb_delta_t<ND>(e, shift, pa, pb, d);
            const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            const float rinv = r2 > 0.f ? rsqrtf(r2) : 0.f;
            const float r = r2 * rinv;
            const float hb = pb.w, ihb = xb.w;
            const float ihn2b = powi<ND>(ihb) * ihb * ihb;
            const float qa = r * iha, qb = r * ihb;
            /* gradW: dr*F(q,h), F = ihn2*dK/dq/q, 1/q = h/r */
            const float Fa = qa != 0.f ? ihn2a * wdK32(qa, wcon) * (ha * rinv) : 0.f;
            const float Fb = qb != 0.f ? ihn2b * wdK32(qb, wcon) * (hb * rinv) : 0.f;
            float cA, cB, cM;  /* gA = d*cA, gB = d*cB, 0.5(gA+gB) = d*cM (times Omega_a with VAR_H) */
            if (var_h) {
                cA = Fa;
                cB = Fb;
                cM = 0.5f * (cA + cB);
                if (is_sph_or_sphb(tb)) om.add(vb.w * (ihna * (-qa * wdK32(qa, wcon) * iha) - pd_coef * wK32(qa, wcon)));
            } else {
                cA = cB = cM = 0.5f * (Fa + Fb);
            }
            /* corrected gradients: vectors gA, gB and their mean (times Omega_a with VAR_H) */
            float gAv[3] = {0.f, 0.f, 0.f}, gBv[3] = {0.f, 0.f, 0.f}, gMv[3] = {0.f, 0.f, 0.f};
            if constexpr (CG) {
                float wa[ND], wb[ND];
                cgw.apply(d, Fa, wa);
                cgw.apply(d, Fb, wb);
#pragma unroll
                for (int k = 0; k < ND; k++) {
                    gAv[k] = var_h ? wa[k] : 0.5f * (wa[k] + wb[k]);
                    gBv[k] = var_h ? wb[k] : 0.5f * (wa[k] + wb[k]);
                    gMv[k] = 0.5f * (gAv[k] + gBv[k]);
                }
            }
            const float densb = xb.x, mb = fabsf(vb.w);
            const float hav = 0.5f * (ha + hb);
            const float dv0 = va.x - vb.x, dv1 = va.y - vb.y, dv2 = va.z - vb.z;
            if (sph && tb != T_DEM && tb != T_DEMB) {
                const float vdr = d[0] * dv0 + d[1] * dv1 + d[2] * dv2;
                float vsig = 0.f;
                if (visc == SPHDEM_VISC_MORRIS) {
                    /* mb visc dg / (r^2 + 0.01 hav^2) with visc = num / (rho_a rho_b):
                     * one division, by the fast reciprocal (2 ulp) */
                    const float num = c.liq_dem() ? liq_visc : visc_nu * (densa + densb);
                    const float dg = CG ? d[0] * gMv[0] + d[1] * gMv[1] + d[2] * gMv[2] : r2 * cM;
                    const float sc = __fdividef(mb * num * dg, (densa * densb) * (r2 + 0.01f * hav * hav));
                    const float dvv[3] = {dv0, dv1, dv2};
#pragma unroll
                    for (int k = 0; k < ND; k++) fv[k].add(dvv[k] * sc);
                } else if (visc == SPHDEM_VISC_MONAGHAN) {
                    const float viss = vdr * rinv;
                    if (!c.liq_dem()) vsig = 2.f * c0 + 2.f * fabsf(viss);
                    const float sv = mb * (viss * vsig * alpha_mon / (densa + densb));
                    const float sc = sv * cM;
#pragma unroll
                    for (int k = 0; k < ND; k++) fv[k].add(CG ? sv * gMv[k] : sc * d[k]);
                } else if (visc == SPHDEM_VISC_ARTIFICIAL) {
                    if (vdr < 0.f) {
                        const float viss = vdr * rinv;
                        const float avsig = 2.f * c0 - 4.f * viss;
                        const float sv = mb * (viss * avsig * alpha_art / (densa + densb));
                        const float sc = sv * cM;
#pragma unroll
                        for (int k = 0; k < ND; k++) fa[k].add(CG ? sv * gMv[k] : sc * d[k]);
                        vsig = fmaxf(vsig, avsig);
                    }
                }
                /* the viscous bound vdc hav^2 / nu increases with hav, and so
                 * does the Courant bound 0.6 hav / vsig under Morris viscosity
                 * (vsig = 2 c0 for every pair): the loop's smallest hav gives
                 * them, bit for bit */
                hmin = fminf(hmin, hav);
                if (visc != SPHDEM_VISC_MORRIS) ndt = fminf(ndt, 0.6f * hav / vsig);
            }
            if (is_boundary(tb)) {
                float fbx[3] = {0.f, 0.f, 0.f};
                boundary32<ND>(cp, NB, b, d[0], d[1], d[2], r, dv0, dv1, dv2, ma, mb, fbx);
#pragma unroll
                for (int k = 0; k < ND; k++) fb[k].add(fbx[k]);
            } else if (tb == T_SPH || tb == T_SPHB) {
                const float pdr2b = xb.y;
                float antic = 0.f;
                if (anti) {
                    const float kdw = wK32(r / hav, wcon) * k_anti_inv;
                    antic = 0.01f * fabsf(pdr2a + pdr2b) * (kdw * kdw) * (kdw * kdw);
                }
                const float pc = pdr2a * cA + pdr2b * cB;
#pragma unroll
                for (int k = 0; k < ND; k++)
                    fp[k].add(CG ? -mb * (pdr2a * gAv[k] + pdr2b * gBv[k]) : -mb * (pc * d[k]));
                if (anti) fq.add(-mb * antic);
            }
        }
        if (hmin < FLT_MAX) {
            if (visc == SPHDEM_VISC_MORRIS) {
                const float vsig = 2.f * c0;
                ndt = fminf(ndt, 0.6f * hmin / vsig);
            }
            ndt = fminf(ndt, vdc * hmin * hmin / visc_nu);
        }
        float roma = 1.f;
        if (var_h) {
            /* Omega = 1 + h*sum/(rho*NDIM): an O(1) number, FP32 is ample */
            const float omega = 1.f + ha * om.s / (densa * ND);
            s.row(FD_OMEGA)[a] = omega;
            roma = 1.f / omega;
        }
        float fsum2 = 0.f;
#pragma unroll
        for (int k = 0; k < ND; k++) {
            const float fpk = fp[k].s * roma + fq.s, fvk = fv[k].s * roma, fak = fa[k].s * roma;
            s.row(FD_FP + k)[a] += fpk;
            s.row(FD_FV + k)[a] += fvk;
            s.row(FD_FB + k)[a] += fb[k].s;
            double *f = s.row(FD_F + k);
            const double fk = f[a] + (double)((fak + fvk) + (fb[k].s + fpk));
            f[a] = fk;
            const float fkf = (float)fk;
            fsum2 += fkf * fkf;
        }
        /* accelCondition (sph.h:566-568), a dt bound: FP32 */
        ndt = fminf(ndt, 0.25f * sqrtf(ha * rsqrtf(fsum2)));
    }
    block_min_atomic(ndt, &g->new_dt_bits);
}

template <int ND, bool CG, bool TILE>
__global__ void __launch_bounds__(BLK) k_dddt(DevCfg c, DevState s, const DevGlobals *__restrict__ g,
                                              const float4 *__restrict__ P0, const float4 *__restrict__ P1,
                                              const float4 *__restrict__ P2,
                                              const int *__restrict__ tg, const int *__restrict__ nbr,
                                              const int *__restrict__ ncnt, int64_t ld, int64_t n,
                                              const double *__restrict__ cgrows,
                                              const int *__restrict__ start, const int *__restrict__ skey) {
    const float4 *shift = stencil_shifts(c, g);
    const bool var_h = c.var_h();
    extern __shared__ float4 st_smem[];
    Staged st = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, false};
    if constexpr (TILE) {
        const int n_t = start[g->n_sph_cells];
        const int64_t a0 = blockIdx.x * (int64_t)blockDim.x;
        if (a0 >= n_t) return;  /* no list owner in this block */
        st = stage_neighbours<ND, 2, 1>(c, const_cast<DevGlobals *>(g), start, skey, P0, P1, P2, a0, n_t, st_smem);
        if (!st.ok) return;
    }
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(tg[a] & 0xff)) return;
    const float wcon = (float)c.wcon;
    const float4 pa = P0[a], va = P1[a];
    const float ha = pa.w, iha = P2[a].w;
    const float ihn2a = powi<ND>(iha) * iha * iha;
    /* VAR_H_CORRECTION: the continuity sum carries 1/Omega_a only, so
     * Omega_a is summed in this loop and applied once at the end */
    const float ihna = powi<ND>(iha), pd_coef = ND * ihna * iha;
    Plain om;
    om.init(-va.w * pd_coef * wK32(0.f, wcon));
    Kahan acc;
    acc.init(0.f);
    Cg32<ND> cgw;
    if constexpr (CG) cgw.load(cgrows, s.cap, a);
    const int cnt = ncnt[a];
    /* 8 entries at a time from the particle's list tiles (two int4 loads) */
    const int4 *tile = reinterpret_cast<const int4 *>(nbr + nl_at(a, 0, ld));
    int4 q0 = make_int4(-1, -1, -1, -1), q1 = q0;
#pragma unroll 2
    for (int j = 0; j < cnt; j++) {
        if ((j & 7) == 0) {
            q0 = __ldg(tile + (j >> 3) * 64);
            q1 = __ldg(tile + (j >> 3) * 64 + 1);
        }
        const int e = q0.x;
        q0 = make_int4(q0.y, q0.z, q0.w, q1.x);
        q1 = make_int4(q1.y, q1.z, q1.w, -1);
        if (e < 0) continue;
        const int b = e & B_MASK;
        float4 pb, vb;
        if constexpr (TILE) {
            const int sl = st_slot<ND>(e >> B_BITS);
            const int off = b - st.lo[sl];
            if ((unsigned)off < (unsigned)st.num[sl]) {
                pb = st.S0[st.base[sl] + off];
                vb = st.S1[st.base[sl] + off];
            } else {
                pb = P0[b];
                vb = P1[b];
            }
        } else {
            pb = P0[b];
            vb = P1[b];
        }
        /* sph / sphBoundary unless the packed mass is negative */
        const int tb = vb.w < 0.f ? (tg[b] & 0xff) : T_SPH;
        const float mb = fabsf(vb.w);
        float d[3];
        nb_delta_t<ND>(e, shift, pa, pb, d);
        const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const float rinv = r2 > 0.f ? rsqrtf(r2) : 0.f;
        const float r = r2 * rinv;
        const float qa = r * iha;
        const float Fa = qa != 0.f ? ihn2a * wdK32(qa, wcon) * (ha * rinv) : 0.f;
        float F, Fb = 0.f;
        if (var_h) {
            F = Fa;
            if (is_sph_or_sphb(tb)) om.add(mb * (ihna * (-qa * wdK32(qa, wcon) * iha) - pd_coef * wK32(qa, wcon)));
        } else {
            const float ihb = P2[b].w;
            const float qb = r * ihb;
            Fb = qb != 0.f ? powi<ND>(ihb) * ihb * ihb * wdK32(qb, wcon) * (pb.w * rinv) : 0.f;
            F = 0.5f * (Fa + Fb);
        }
        const float dv[3] = {va.x - vb.x, va.y - vb.y, va.z - vb.z};
        float vdr;
        if constexpr (CG) {
            /* corrected gradient of a (and of b's kernel) applied with a's invM */
            float wa[ND], wb[ND];
            cgw.apply(d, Fa, wa);
            if (!var_h) cgw.apply(d, Fb, wb);
            vdr = 0.f;
#pragma unroll
            for (int k = 0; k < ND; k++) vdr += dv[k] * (var_h ? wa[k] : 0.5f * (wa[k] + wb[k]));
            F = 1.f;
        } else {
            vdr = dv[0] * d[0] + dv[1] * d[1] + dv[2] * d[2];
        }
        if (!(is_boundary(tb) || tb == T_DEM)) acc.add(mb * vdr * F);
    }
    float roma = 1.f;
    if (var_h) {
        const float omega = 1.f + ha * om.s / (P2[a].x * ND);
        s.row(FD_OMEGA)[a] = omega;
        roma = 1.f / omega;
    }
    s.row(FD_DDDT)[a] += (double)(acc.s * roma);
}

/* total += sum of x */
__global__ void k_sum(int64_t n, const int *__restrict__ x, int *total) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int v = __reduce_add_sync(0xffffffffu, i < n ? x[i] : 0);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(total, v);
}

/* rows of the neighbour list in tag order (count pass when idx == nullptr) */
__global__ void k_list_export(DevState s, const int *tg, const int *nbr, const int *ncnt, int64_t ld, int64_t n,
                              int *cnt, const long long *offs, int *idx) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (a >= n) return;
    if (!is_sph_or_sphb(tg[a] & 0xff)) return;
    const int tag = s.irow(FI_TAG)[a];
    const int m = ncnt[a];
    if (!idx) {
        int v = 0;
        for (int j = 0; j < m; j++) v += nbr[nl_at(a, j, ld)] >= 0;
        cnt[tag] = v;
        return;
    }
    int k = 0;
    for (int j = 0; j < m; j++) {
        const int e = nbr[nl_at(a, j, ld)];
        if (e >= 0) idx[offs[tag] + k++] = s.irow(FI_TAG)[e & B_MASK];
    }
}

/* The list rows of the SPH/SPHB particles as the adjoint's per-step pair
 * tables, in tag space: nb[slot * cap + off + k] = tag_b | shift << 26 (shift
 * = (sh_x + 1) | (sh_y + 1) << 2 | (sh_z + 1) << 4, the periodic image of b),
 * oc[slot * n + tag_a] = (off, count).  One atomic per warp reserves the
 * warp's entries; an overflowing particle records count 0 and the caller sees
 * cnt[slot] > cap. */
template <int ND>
__global__ void k_adj_pairs(DevState s, const DevGlobals *__restrict__ g, const int *__restrict__ skey,
                            const int *__restrict__ tg, const int *__restrict__ nbr, const int *__restrict__ ncnt,
                            int64_t ld, int64_t n, int *nb, int2 *oc, int *cnt, int64_t cap,
                            const int *__restrict__ slot) {
    const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool live = a < n && is_sph_or_sphb(tg[a] & 0xff);
    const int m = live ? ncnt[a] : 0;
    int k = 0;
    for (int j = 0; j < m; j++) k += nbr[nl_at(a, j, ld)] >= 0;
    const int lane = threadIdx.x & 31;
    int incl = k;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int js = *slot;
    int base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(cnt + js, total);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (!live) return;
    const int64_t off = (int64_t)base + incl - k;
    const int64_t room = cap - off;
    int *out = nb + (int64_t)js * cap + off;
    const int dims[3] = {g->sdims[0], g->sdims[1], g->sdims[2]};
    int cc[3] = {0, 0, 0};
    decode<ND>(skey[a], dims, cc);
    int q = 0;
    for (int j = 0; j < m && q < room; j++) {
        const int e = nbr[nl_at(a, j, ld)];
        if (e < 0) continue;
        int o[3];
        nl_decode_code(e >> B_BITS, o);
        int code = 0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            int sh = 0;
            if (d < ND) {
                const int t = cc[d] + o[d];
                sh = t < 0 ? -1 : (t >= dims[d] ? 1 : 0);
            }
            code |= (sh + 1) << (2 * d);
        }
        out[q++] = s.irow(FI_TAG)[e & B_MASK] | (code << B_BITS);
    }
    oc[(int64_t)js * n + s.irow(FI_TAG)[a]] = make_int2((int)off, room >= k ? k : 0);
}

/* list build: grid-stride over 32-particle slices, one wave of resident blocks */
template <int ND, bool COUNT, int G>
int nlist_blocks(int64_t particles) {
    static int resident = 0;
    if (!resident) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_nlist<ND, COUNT, G>, NL_WARPS * 32, 0);
        resident = std::max(1, sms * per_sm);
    }
    const int per_block = 32 / G * NL_WARPS;
    const int64_t need = (particles + per_block - 1) / per_block;
    return (int)std::max<int64_t>(1, std::min<int64_t>(resident, need));
}

}  // namespace

void mixed_list_export(sphdem_ctx *c, int *cnt, const long long *offs, int *idx) {
    k_list_export<<<grid_for(c->n, 256), 256, 0, c->stream>>>(c->A, c->mx_tg, c->mx_nbr, c->mx_ncnt, (int64_t)c->mx_maxn, c->n,
                                                              cnt, offs, idx);
}

void mixed_adj_pairs(sphdem_ctx *c, int *nb, int2 *oc, int *cnt, int64_t cap, const int *slot) {
    const int g = grid_for(c->n, 128);
    if (c->cfg.nd == 3)
        k_adj_pairs<3><<<g, 128, 0, c->stream>>>(c->A, c->g, c->buf.skey, c->mx_tg, c->mx_nbr, c->mx_ncnt, (int64_t)c->mx_maxn,
                                                 c->n, nb, oc, cnt, cap, slot);
    else if (c->cfg.nd == 2)
        k_adj_pairs<2><<<g, 128, 0, c->stream>>>(c->A, c->g, c->buf.skey, c->mx_tg, c->mx_nbr, c->mx_ncnt, (int64_t)c->mx_maxn,
                                                 c->n, nb, oc, cnt, cap, slot);
    else
        k_adj_pairs<1><<<g, 128, 0, c->stream>>>(c->A, c->g, c->buf.skey, c->mx_tg, c->mx_nbr, c->mx_ncnt, (int64_t)c->mx_maxn,
                                                 c->n, nb, oc, cnt, cap, slot);
}

/* ---------------------------------------------------------------------- */

namespace mixed {

void pack(sphdem_ctx *c, bool middle) {
#define L_(ND)                                                                                                  \
    SPHDEM_LAUNCH(c, "pack32", k_pack<ND>, grid_for(c->n, 256), 256, 0, c->cfg, c->A, c->buf.skey, c->g,         \
                  c->mx_pos, c->mx_vel, c->mx_aux, c->mx_tg, (int)middle, c->mx_ds, c->mx_nb, c->n)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
}

void nlist(sphdem_ctx *c, int depth, bool soft) {
    /* below these counts the warps of 32 particles do not fill the chip and the
     * pass is the length of one warp's chain.  Two builds, one / four lanes per
     * particle: 2D 6.5k 38 / 26 us, 23k 45 / 30, 44k 46 / 38, 86k 50 / 56; 3D
     * 3.8k 112 / 69, 23k 113 / 82, 47k 123 / 131, 91k 153 / 228 */
    const bool split = c->n < (c->cfg.nd == 3 ? 40000 : 65000);
#define LG_(ND, G)                                                                                              \
    SPHDEM_LAUNCH(c, "nlist32", (k_nlist<ND, false, G>),                                                       \
                  (std::max(1, nlist_blocks<ND, false, G>(c->n) / c->grid_div)), NL_WARPS * 32, 0, c->cfg, c->dcfg, \
                  c->A, c->buf.start, c->buf.skey, c->g, c->mx_pos, c->mx_tg, c->mx_nbr, c->mx_ncnt, depth,      \
                  (int)soft, c->mx_bandn)
#define L_(ND)            \
    do {                  \
        if (split)        \
            LG_(ND, 4);   \
        else              \
            LG_(ND, 1);   \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LG_
}

/* neighbour counts of the current buckets and records, into scratch of the
 * rebuild: mx_ncnt holds the counts of the lists that are there.  Candidates FP32
 * cannot decide and the particle itself count as neighbours, so these are upper
 * bounds */
static int *nlist_count(sphdem_ctx *c) {
    int *cnt = c->buf.slot;
    SPHDEM_CUDA_CHECK(cudaMemsetAsync(cnt, 0, c->n * sizeof(int), c->stream));
#define L_(ND)                                                                                                    \
    k_nlist<ND, true, 1><<<nlist_blocks<ND, true, 1>(c->n), NL_WARPS * 32, 0, c->stream>>>(                           \
        c->cfg, c->dcfg, c->A, c->buf.start, c->buf.skey, c->g, c->mx_pos, c->mx_tg, nullptr,        \
        cnt, 0, 0, nullptr)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
    SPHDEM_CUDA_CHECK(cudaGetLastError());
    return cnt;
}

void nlist_pairs(sphdem_ctx *c, int *total) {
    if (c->cfg.precision == SPHDEM_PREC_MIXED) pack(c, false);
    else pack_positions(c, false);
    k_sum<<<grid_for(c->n, 256), 256, 0, c->stream>>>(c->n, nlist_count(c), total);
    SPHDEM_CUDA_CHECK(cudaGetLastError());
}

int nlist_max_count(sphdem_ctx *c) {
    const int *cnt = nlist_count(c);
    std::vector<int> h(c->n);
    SPHDEM_CUDA_CHECK(cudaMemcpyAsync(h.data(), cnt, c->n * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SPHDEM_CUDA_CHECK(cudaStreamSynchronize(c->stream));
    int m = 0;
    for (int v : h) m = std::max(m, v);
    return m;
}

void eos(sphdem_ctx *c) {
    SPHDEM_LAUNCH(c, "eos32", k_eos32, grid_for(c->n, c->blk_pair), c->blk_pair, 0, c->cfg, c->A, c->mx_aux, c->mx_tg, c->n);
}

void force(sphdem_ctx *c) {
    if (force_lists(c)) return;
    const double *cgrows = corrected_gradient(c) ? c->cg : nullptr;
    /* neighbour records staged through shared memory (2D and 3D) */
    const bool tile = c->cfg.nd > 1 && c->force_tile;
    const size_t st_bytes = tile ? (size_t)3 * ST_CAP * sizeof(float4) : 0;
#define LP_(ND, P, T)                                                                                           \
    SPHDEM_LAUNCH(c, "force32", (k_force<ND, P, T>), grid_for(c->n, c->blk_pair), c->blk_pair, st_bytes, c->cfg, \
                  c->dcfg, c->A, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_tg, c->mx_nbr,         \
                  c->mx_ncnt, (int64_t)c->mx_maxn, c->n, c->mx_nb, cgrows, c->buf.start, c->buf.skey)
#define L_(ND)                              \
    do {                                    \
        if (cgrows && tile)                 \
            LP_(ND, PHYS_CG, true);         \
        else if (cgrows)                    \
            LP_(ND, PHYS_CG, false);        \
        else if (tile)                      \
            LP_(ND, PHYS_GENERIC, true);    \
        else                                \
            LP_(ND, PHYS_GENERIC, false);   \
    } while (0)
    SPHDEM_ND_DISPATCH(c->cfg.nd, L_);
#undef L_
#undef LP_
}

/* Kernel attributes the step needs, set once per process outside any
 * stream capture: the dynamic shared memory of the staged force passes. */
void prepare(sphdem_ctx *) {
    static bool done = false;
    if (done) return;
    const int bytes = (int)(3 * ST_CAP * sizeof(float4));
#define A_(ND, P) \
    SPHDEM_CUDA_CHECK(cudaFuncSetAttribute(k_force<ND, P, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))
    A_(2, PHYS_GENERIC);
    A_(2, PHYS_CG);
    A_(3, PHYS_GENERIC);
    A_(3, PHYS_CG);
#undef A_
    const int bytes2 = (int)(2 * ST_CAP * sizeof(float4));
#define D_(ND) \
    SPHDEM_CUDA_CHECK(cudaFuncSetAttribute(k_dddt<ND, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes2))
    D_(2);
    D_(3);
#undef D_
    prepare_lists();
    done = true;
}

void dddt(sphdem_ctx *c) {
    if (dddt_lists(c)) return;
    /* CORRECTED_GRADIENT, or 1D */
    const double *cgrows = corrected_gradient(c) ? c->cg : nullptr;
    const bool tile = c->cfg.nd > 1 && c->force_tile;
    const size_t st_bytes = tile ? (size_t)2 * ST_CAP * sizeof(float4) : 0;
#define LD_(ND, CGF, T)                                                                                         \
    SPHDEM_LAUNCH(c, "dddt32", (k_dddt<ND, CGF, T>), grid_for(c->n, c->blk_pair), c->blk_pair, st_bytes,   \
                  c->cfg, c->A, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_tg, c->mx_nbr,          \
                  c->mx_ncnt, (int64_t)c->mx_maxn, c->n, cgrows, c->buf.start, c->buf.skey)
    if (c->cfg.nd == 1) {
        if (cgrows)
            LD_(1, true, false);
        else
            LD_(1, false, false);
    } else if (c->cfg.nd == 2) {
        if (tile)
            LD_(2, true, true);
        else
            LD_(2, true, false);
    } else {
        if (tile)
            LD_(3, true, true);
        else
            LD_(3, true, false);
    }
#undef LD_
}

}  // namespace mixed
}  // namespace sphdem
