/*
 * Force and continuity passes over the neighbour lists, specialised on the
 * physics class so that the unused viscosity forms, accumulators and branches
 * compile away: Morris viscosity with and without VAR_H_CORRECTION (the
 * coupled sedimentation) and artificial viscosity with constant h (the dam
 * break), no anticlumping, in 2D and 3D.  Everything else runs the general
 * passes of pairs32.cu.
 *
 * Both passes are bound by their gathers (L1 wavefronts half of the peak, 85 % of
 * the sectors from L1, waits for them the largest stall) and by issue next to
 * it, not by DRAM.  So a lane takes two list entries at a time and does their
 * arithmetic in packed FP32 (f32x2: two results per issued instruction), with
 * one Kahan sum for the even and one for the odd entries; the Wendland gradient is taken in its closed form
 * F(r, h) = -10 C / h^(d+2) (2 - r/h)^3, which needs neither dK/dq / q nor a
 * case for r = 0; types other than sph / sphBoundary, which the sign of the
 * packed mass marks, leave the main path.  G consecutive lanes share a
 * particle and take its groups of 8 entries in turn, their sums joined at the
 * end with the rounding errors kept: small populations fill the chip with
 * G > 1 (rules: force_lanes, dddt_lanes).  Before / now, us: coupled force pass
 * of 1.08 M particles 1136 / 732, continuity 533 / 407; of 3,768 particles 115 /
 * 27 and 64 / 14; dam break of 23,018 26 / 14 and 19 / 12.
 */
#include <type_traits>

#include "mixed.cuh"

namespace sphdem {
namespace {

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

/* 1/sqrt(x) of x > 0 (2 ulp), flushing denormals */
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* 1/x of a normal x > 0 (1 ulp) */
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* Geometry of a lane's particle and two of its list entries: displacement,
 * 1/r (finite at r = 0), r, and (2 - r/h_a)^3 cut at 0. */
template <int ND>
struct Duo {
    float2 d[ND], r2, ri, r, t3;
    __device__ __forceinline__ void set(float4 pa, float4 p0, float4 p1, float4 s0, float4 s1, float2 niha) {
        d[0] = make_float2(pa.x - p0.x - s0.x, pa.x - p1.x - s1.x);
        r2 = __fmul2_rn(d[0], d[0]);
        if constexpr (ND > 1) {
            d[1] = make_float2(pa.y - p0.y - s0.y, pa.y - p1.y - s1.y);
            r2 = __ffma2_rn(d[1], d[1], r2);
        }
        if constexpr (ND > 2) {
            d[2] = make_float2(pa.z - p0.z - s0.z, pa.z - p1.z - s1.z);
            r2 = __ffma2_rn(d[2], d[2], r2);
        }
        ri = make_float2(rsqrt_ftz(fmaxf(r2.x, 1e-37f)), rsqrt_ftz(fmaxf(r2.y, 1e-37f)));
        r = __fmul2_rn(r2, ri);
        float2 t = __ffma2_rn(r, niha, both(2.f));
        t = make_float2(fmaxf(t.x, 0.f), fmaxf(t.y, 0.f));
        t3 = __fmul2_rn(__fmul2_rn(t, t), t);
    }
};

/* One pair by the general passes' own expressions (pairs32.cu): the kernel
 * gradient in its expanded form, which the 8-lane passes of the coupled case take.
 * It is neither faster (3,768 particles: force 26.7 us a launch against 23.0 in the
 * closed form, continuity 14.1 against 11.7) nor nearer to FP64: it keeps the
 * results of small boxes where they have been.  In those a few stiff spheres amplify
 * a rounding within ten steps, and the closed form moves the paths by 0.4e-9 to
 * 1.1e-9 of the box, as far as either form is from FP64 (0.9e-9 to 1.6e-9). */
template <int ND>
struct PlainPair {
    float d[3], r2, r, rinv;
    __device__ __forceinline__ void set(int e, const float4 *shift, float4 pa, float4 pb) {
        nb_delta_t<ND>(e, shift, pa, pb, d);
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        rinv = r2 > 0.f ? rsqrtf(r2) : 0.f;
        r = r2 * rinv;
    }
    __device__ __forceinline__ float gradient(float h, float ih, float wcon) const {
        const float ihn2 = powi<ND>(ih) * ih * ih, q = r * ih;
        return q != 0.f ? ihn2 * wdK32(q, wcon) * (h * rinv) : 0.f;
    }
};

/* d/dh of the kernel at b, W_h = C (10 q^2 - d t (1 + 2q)) t^3 / h^(d+1) with
 * t = 2 - q cut at 0 (calcOmega, sph.h:438-451), without C / h^(d+1) */
template <int ND>
__device__ __forceinline__ float2 omega_poly(float2 q, float2 t3) {
    const float2 u = __ffma2_rn(q, both(10.f + 2.f * ND), both(-3.f * ND));
    return __fmul2_rn(__ffma2_rn(u, q, both(-2.f * ND)), t3);
}

/* visit a lane's share of a particle's list: body(std::bool_constant masked,
 * e0, e1), two entries at a time, the lane's next group of 8 in flight.  In a
 * masked call the second entry may be < 0 (none). */
template <int G, class Body>
__device__ __forceinline__ void visit_list(const int *__restrict__ nbr, int64_t a, int64_t ld, int cnt, int sub, Body &&body) {
    const int4 *tile = reinterpret_cast<const int4 *>(nbr + nl_at(a, 0, ld));
    int4 n0 = make_int4(-1, -1, -1, -1), n1 = n0;
    if (sub * 8 < cnt) {
        n0 = __ldg(tile + sub * 64);
        n1 = __ldg(tile + sub * 64 + 1);
    }
    for (int gi = sub; gi * 8 < cnt; gi += G) {
        const int4 c0 = n0, c1 = n1;
        if ((gi + G) * 8 < cnt) {
            n0 = __ldg(tile + (gi + G) * 64);
            n1 = __ldg(tile + (gi + G) * 64 + 1);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = cnt - gi * 8 - h * 4;
            int4 e = h ? c1 : c0;
            if (m >= 4) {
                body(std::false_type{}, e.x, e.y);
                body(std::false_type{}, e.z, e.w);
            } else if (m > 0) {
                /* the list's last entries: what follows them is not read */
                if (m < 2) e.y = -1;
                if (m < 3) e.z = -1;
                body(std::true_type{}, e.x, e.y);
                if (m > 2) body(std::true_type{}, e.z, -1);
            }
        }
    }
}

/* The middle phase's calcForce (sphIncompress.h:899-972) with calcOmega and
 * the Courant / viscous / acceleration time-step bounds. */
template <int ND, int VISC, bool VARH, int G, bool TILE>
__global__ void __launch_bounds__(BLK, 4) k_force_list(DevCfg c, const DevCfg *__restrict__ cp, DevState s,
                                                    DevGlobals *__restrict__ g, const float4 *__restrict__ P0,
                                                    const float4 *__restrict__ P1, const float4 *__restrict__ P2,
                                                    const int *__restrict__ tg,
                                                    const int *__restrict__ nbr, const int *__restrict__ ncnt,
                                                    int64_t ld, int64_t n, const float4 *__restrict__ NB,
                                                    const int *__restrict__ start, const int *__restrict__ skey) {
    const float4 *shift = stencil_shifts(c, g);
    extern __shared__ float4 st_smem[];
    Staged st = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, false};
    if constexpr (TILE) {
        const int n_t = start[g->n_sph_cells];
        const int64_t a0 = blockIdx.x * (int64_t)(blockDim.x / G);
        if (a0 >= n_t) return; /* no list owner in this block */
        st = stage_neighbours<ND, 3, G>(c, g, start, skey, P0, P1, P2, a0, n_t, st_smem);
        if (!st.ok) return;
    }
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const int ta = a < n ? (tg[a] & 0xff) : -1;
    const bool act = is_sph_or_sphb(ta);
    float4 pa = make_float4(0.f, 0.f, 0.f, 1.f), va = pa, xa = pa;
    if (act) {
        pa = P0[a];
        va = P1[a];
        xa = P2[a];
    }
    const float ha = pa.w, iha = xa.w, densa = xa.x, pdr2a = xa.y, cFa = xa.z;
    const float c0 = (float)c.spsound, visc_nu = (float)c.viscosity;
    const float liq_visc = (float)(2.0 * c.viscosity * c.dens);
    const bool liq = c.liq_dem();
    Kahan2 fp[ND], fv[ND];   /* fv: viscous force; of artificial viscosity, which f alone takes */
    Kahan fb[ND];
    bool wall = false;       /* a repulsive boundary particle among the neighbours */
#pragma unroll
    for (int k = 0; k < ND; k++) {
        fp[k].init();
        fv[k].init();
        fb[k].init(0.f);
    }
    float2 om = both(0.f);
    float hmin = FLT_MAX;  /* smallest hav of the fluid pairs */
    float hbest = FLT_MAX, vbest = 1.f; /* the pair with the smallest hav / vsig (artificial viscosity) */
    const float2 niha = both(-iha);
    constexpr bool EXPANDED = G == 8 && VISC == SPHDEM_VISC_MORRIS;
    const float wcon = (float)c.wcon;
    auto fetch = [&](int e, float4 &p, float4 &v, float4 &x) {
        const int b = e & B_MASK;
        if constexpr (TILE) {
            const int sl = st_slot<ND>(e >> B_BITS);
            const int off = b - st.lo[sl];
            if ((unsigned)off < (unsigned)st.num[sl]) {
                const int k = st.base[sl] + off;
                p = st.S0[k];
                v = st.S1[k];
                x = st.S2[k];
                return;
            }
        }
        p = P0[b];
        v = P1[b];
        x = P2[b];
    };
    auto body = [&](auto masked, int e0, int e1) {
        constexpr bool MASK = decltype(masked)::value;
        /* an entry that is none stands for the particle itself without mass */
        const int self_e = (int)a | (13 << B_BITS);
        const bool none1 = MASK && e1 < 0;
        if (none1) e1 = self_e;
        float4 p0, v0, x0, p1, v1, x1;
        fetch(e0, p0, v0, x0);
        fetch(e1, p1, v1, x1);
        Duo<ND> q;
        q.set(pa, p0, p1, shift[e0 >> B_BITS], shift[e1 >> B_BITS], niha);
        if (none1) v1.w = 0.f;
        /* masses in the viscous term, and in the terms of sph / sphBoundary only */
        float mv0 = v0.w, mv1 = v1.w;
        float hav0 = 0.5f * (ha + p0.w), hav1 = 0.5f * (ha + p1.w);
        const float2 hav = make_float2(hav0, hav1);
        float2 dv[3];
        dv[0] = make_float2(va.x - v0.x, va.x - v1.x);
        dv[1] = make_float2(va.y - v0.y, va.y - v1.y);
        dv[2] = make_float2(va.z - v0.z, va.z - v1.z);
        if (none1) hav1 = FLT_MAX;
        if (fminf(mv0, mv1) < 0.f) {
            /* walls act by the viscous term here and by their own force below */
            if (mv0 < 0.f) {
                const int tb = tg[e0 & B_MASK] & 0xff;
                wall |= is_boundary(tb);
                mv0 = tb == T_DEM || tb == T_DEMB ? 0.f : -mv0;
                if (mv0 == 0.f) hav0 = FLT_MAX;
            }
            if (mv1 < 0.f) {
                const int tb = tg[e1 & B_MASK] & 0xff;
                wall |= is_boundary(tb);
                mv1 = tb == T_DEM || tb == T_DEMB ? 0.f : -mv1;
                if (mv1 == 0.f) hav1 = FLT_MAX;
            }
        }
        const float2 m = make_float2(fmaxf(v0.w, 0.f), fmaxf(v1.w, 0.f));
        const float2 mv = make_float2(mv0, mv1);
        /* F of b's kernel, cut at 2 h_b */
        float2 tb = make_float2(fmaxf(fmaf(q.r.x, -x0.w, 2.f), 0.f), fmaxf(fmaf(q.r.y, -x1.w, 2.f), 0.f));
        tb = __fmul2_rn(__fmul2_rn(tb, tb), tb);
        float2 Fb = make_float2(x0.z * tb.x, x1.z * tb.y);
        float2 Fa = __fmul2_rn(q.t3, both(cFa));
        if constexpr (EXPANDED) {
            PlainPair<ND> u0, u1;
            u0.set(e0, shift, pa, p0);
            u1.set(e1, shift, pa, p1);
            Fa = make_float2(u0.gradient(ha, iha, wcon), u1.gradient(ha, iha, wcon));
            Fb = make_float2(u0.gradient(p0.w, x0.w, wcon), u1.gradient(p1.w, x1.w, wcon));
        }
        const float2 cM = __fmul2_rn(__fadd2_rn(Fa, Fb), both(0.5f)); /* 0.5 (gA + gB) = d cM */
        float2 pc;
        if constexpr (VARH) {
            if constexpr (EXPANDED) {
                pc = make_float2(pdr2a * Fa.x + x0.y * Fb.x, pdr2a * Fa.y + x1.y * Fb.y);
            } else {
                pc = make_float2(x0.y * Fb.x, x1.y * Fb.y);
                pc = __ffma2_rn(both(pdr2a), Fa, pc);
            }
            om = __ffma2_rn(m, omega_poly<ND>(__fmul2_rn(q.r, both(iha)), q.t3), om);
        } else {
            pc = __fmul2_rn(make_float2(pdr2a + x0.y, pdr2a + x1.y), cM);
        }
        const float2 nm = make_float2(-m.x, -m.y);
        if constexpr (EXPANDED) {
#pragma unroll
            for (int k = 0; k < ND; k++) fp[k].add_product(nm, __fmul2_rn(pc, q.d[k]));
        } else {
            pc = __fmul2_rn(pc, nm);
#pragma unroll
            for (int k = 0; k < ND; k++) fp[k].add_product(pc, q.d[k]);
        }
        if constexpr (VISC == SPHDEM_VISC_MORRIS) {
            /* m_b visc dg / (r^2 + 0.01 hav^2), visc = num / (rho_a rho_b) */
            float2 num = __fmul2_rn(__fmul2_rn(q.r2, cM), mv);
            num = liq ? __fmul2_rn(num, both(liq_visc))
                      : __fmul2_rn(num, __fmul2_rn(make_float2(densa + x0.x, densa + x1.x), both(visc_nu)));
            const float2 den = __fmul2_rn(__fmul2_rn(both(densa), make_float2(x0.x, x1.x)),
                                          __ffma2_rn(__fmul2_rn(hav, hav), both(0.01f), q.r2));
            const float2 sc = make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
#pragma unroll
            for (int k = 0; k < ND; k++) fv[k].add_product(dv[k], sc);
        } else {
            float2 vdr = __fmul2_rn(q.d[0], dv[0]);
#pragma unroll
            for (int k = 1; k < ND; k++) vdr = __ffma2_rn(q.d[k], dv[k], vdr);
            /* approach speed (<= 0): receding pairs have none */
            const float2 vs = __fmul2_rn(make_float2(fminf(vdr.x, 0.f), fminf(vdr.y, 0.f)), q.ri);
            const float2 sig = __ffma2_rn(vs, both(-4.f), both(2.f * c0));
            const float2 num = __fmul2_rn(__fmul2_rn(__fmul2_rn(vs, sig), __fmul2_rn(mv, both((float)c.alpha_art))), cM);
            /* to the last place, as a division; a dam break's step takes the 0.28 ms
             * it took with bare estimates (full divisions: 0.29) */
            const float2 den = make_float2(densa + x0.x, densa + x1.x);
            const float2 sc = quotient(num, den, make_float2(rcp_ftz(den.x), rcp_ftz(den.y)));
#pragma unroll
            for (int k = 0; k < ND; k++) fv[k].add_product(q.d[k], sc);
            /* hav / vsig < hbest / vbest, without a division */
            if (vs.x < 0.f && hav0 * vbest < hbest * sig.x) {
                hbest = hav0;
                vbest = sig.x;
            }
            if (vs.y < 0.f && hav1 * vbest < hbest * sig.y) {
                hbest = hav1;
                vbest = sig.y;
            }
        }
        hmin = fminf(hmin, fminf(hav0, hav1));
    };
    if (act) visit_list<G>(nbr, a, ld, ncnt[a], sub, body);
    if (wall) {
        /* the repulsive boundary particles among this lane's entries: eight
         * records in flight, then those of walls one by one */
        const int cnt = ncnt[a];
        for (int gi = sub; gi * 8 < cnt; gi += G) {
            unsigned walls = 0u;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int e = gi * 8 + j < cnt ? nbr[nl_at(a, gi * 8 + j, ld)] : (int)a;
                if (P1[e & B_MASK].w < 0.f) walls |= 1u << j;
            }
            for (; walls; walls &= walls - 1) {
                const int e = nbr[nl_at(a, gi * 8 + __ffs(walls) - 1, ld)], b = e & B_MASK;
                if (!is_boundary(tg[b] & 0xff)) continue;
                const float4 pb = P0[b], vb = P1[b];
                float d[3], fbx[3] = {0.f, 0.f, 0.f};
                nb_delta_t<ND>(e, shift, pa, pb, d);
                const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                boundary32<ND>(cp, NB, b, d[0], d[1], d[2], r2 * rsqrt_ftz(fmaxf(r2, 1e-37f)), va.x - vb.x, va.y - vb.y,
                               va.z - vb.z, va.w, -vb.w, fbx);
#pragma unroll
                for (int k = 0; k < ND; k++) fb[k].add(fbx[k]);
            }
        }
    }

    float ndt = FLT_MAX;
    if (ta == T_SPH && hmin < FLT_MAX) {
        /* the viscous bound vdc hav^2 / nu increases with hav, and so does the
         * Courant bound 0.6 hav / vsig under Morris viscosity (vsig = 2 c0) */
        if (VISC == SPHDEM_VISC_MORRIS) ndt = fminf(ndt, 0.6f * hmin / (2.f * c0));
        else if (hbest < FLT_MAX) ndt = fminf(ndt, 0.6f * hbest / vbest);
        ndt = fminf(ndt, 0.125f * hmin * hmin / visc_nu);
    }
    float tp[ND], tv[ND], tb[ND];
#pragma unroll
    for (int k = 0; k < ND; k++) {
        tp[k] = fp[k].template total<G>();
        tv[k] = fv[k].template total<G>();
        tb[k] = fb[k].template total<G>();
    }
    float omt = om.x + om.y;
    if (VARH) {
#pragma unroll
        for (int o = 1; o < G; o <<= 1) omt += __shfl_xor_sync(0xffffffffu, omt, o);
    }
    if (act && sub == 0) {
        float roma = 1.f;
        if (VARH) {
            /* Omega = 1 + h sum / (rho NDIM), the sum with a's own term -m d K(0) / h^(d+1) */
            const float hd1 = powi<ND>(iha) * iha;
            const float sum = hd1 * (omt * wcon - va.w * ND * wK32(0.f, wcon));
            const float omega = 1.f + ha * sum / (densa * ND);
            s.row(FD_OMEGA)[a] = omega;
            roma = 1.f / omega;
        }
        float fsum2 = 0.f;
#pragma unroll
        for (int k = 0; k < ND; k++) {
            /* an sphBoundary particle takes no viscous force */
            const float fpk = tp[k] * roma, fvk = ta == T_SPH ? tv[k] * roma : 0.f;
            s.row(FD_FP + k)[a] += fpk;
            if (VISC == SPHDEM_VISC_MORRIS) s.row(FD_FV + k)[a] += fvk;
            s.row(FD_FB + k)[a] += tb[k];
            double *f = s.row(FD_F + k);
            const double fk = f[a] + (double)(fvk + (tb[k] + fpk));
            f[a] = fk;
            const float fkf = (float)fk;
            fsum2 += fkf * fkf;
        }
        /* accelCondition (sph.h:566-568), a dt bound: FP32 */
        ndt = fminf(ndt, 0.25f * sqrtf(ha * rsqrtf(fsum2)));
    }
    block_min_atomic(ndt, &g->new_dt_bits);
}

/* The end phase's calcDddtDudt (sphIncompress.h:783-851) with calcOmega. */
template <int ND, bool VARH, int G, bool TILE>
__global__ void __launch_bounds__(BLK) k_dddt_list(DevCfg c, DevState s, DevGlobals *__restrict__ g,
                                                   const float4 *__restrict__ P0, const float4 *__restrict__ P1,
                                                   const float4 *__restrict__ P2,
                                                   const int *__restrict__ tg, const int *__restrict__ nbr,
                                                   const int *__restrict__ ncnt, int64_t ld, int64_t n,
                                                   const int *__restrict__ start, const int *__restrict__ skey) {
    const float4 *shift = stencil_shifts(c, g);
    extern __shared__ float4 st_smem[];
    Staged st = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, false};
    if constexpr (TILE) {
        const int n_t = start[g->n_sph_cells];
        const int64_t a0 = blockIdx.x * (int64_t)(blockDim.x / G);
        if (a0 >= n_t) return; /* no list owner in this block */
        st = stage_neighbours<ND, 2, G>(c, g, start, skey, P0, P1, P2, a0, n_t, st_smem);
        if (!st.ok) return;
    }
    const int64_t a = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
    const int sub = threadIdx.x % G;
    const bool act = a < n && is_sph_or_sphb(tg[a] & 0xff);
    float4 pa = make_float4(0.f, 0.f, 0.f, 1.f), va = pa, xa = pa;
    if (act) {
        pa = P0[a];
        va = P1[a];
        xa = P2[a];
    }
    const float ha = pa.w, iha = xa.w;
    const float cFa = xa.y;
    Kahan2 acc;
    acc.init();
    float2 om = both(0.f);
    const float2 niha = both(-iha);
    constexpr bool EXPANDED = G == 8 && VARH;
    const float wcon = (float)c.wcon;
    auto body = [&](auto masked, int e0, int e1) {
        constexpr bool MASK = decltype(masked)::value;
        const bool none1 = MASK && e1 < 0;
        if (none1) e1 = (int)a | (13 << B_BITS);
        const int b0 = e0 & B_MASK, b1 = e1 & B_MASK;
        float4 p0, v0, p1, v1;
        auto fetch = [&](int e, float4 &p, float4 &v) {
            const int b = e & B_MASK;
            if constexpr (TILE) {
                const int sl = st_slot<ND>(e >> B_BITS);
                const int off = b - st.lo[sl];
                if ((unsigned)off < (unsigned)st.num[sl]) {
                    p = st.S0[st.base[sl] + off];
                    v = st.S1[st.base[sl] + off];
                    return;
                }
            }
            p = P0[b];
            v = P1[b];
        };
        fetch(e0, p0, v0);
        fetch(e1, p1, v1);
        Duo<ND> q;
        q.set(pa, p0, p1, shift[e0 >> B_BITS], shift[e1 >> B_BITS], niha);
        if (none1) v1.w = 0.f;
        const float2 mo = make_float2(fmaxf(v0.w, 0.f), fmaxf(v1.w, 0.f));
        float2 m = mo;
        if (fminf(v0.w, v1.w) < 0.f) {
            /* neither sph / sphBoundary nor DEM: repulsive boundary particles and DEM take no part */
            if (v0.w < 0.f) {
                const int tb = tg[b0] & 0xff;
                if (!(is_boundary(tb) || tb == T_DEM)) m.x = -v0.w;
            }
            if (v1.w < 0.f) {
                const int tb = tg[b1] & 0xff;
                if (!(is_boundary(tb) || tb == T_DEM)) m.y = -v1.w;
            }
        }
        float2 vdr = __fmul2_rn(make_float2(va.x - v0.x, va.x - v1.x), q.d[0]);
        if constexpr (ND > 1) vdr = __ffma2_rn(make_float2(va.y - v0.y, va.y - v1.y), q.d[1], vdr);
        if constexpr (ND > 2) vdr = __ffma2_rn(make_float2(va.z - v0.z, va.z - v1.z), q.d[2], vdr);
        float2 F;
        if constexpr (VARH) {
            F = q.t3; /* times cFa / Omega_a at the end */
            om = __ffma2_rn(mo, omega_poly<ND>(__fmul2_rn(q.r, both(iha)), q.t3), om);
            if constexpr (EXPANDED) {
                PlainPair<ND> u0, u1;
                u0.set(e0, shift, pa, p0);
                u1.set(e1, shift, pa, p1);
                F = make_float2(u0.gradient(ha, iha, wcon), u1.gradient(ha, iha, wcon));
                vdr = make_float2((va.x - v0.x) * u0.d[0] + (va.y - v0.y) * u0.d[1] + (va.z - v0.z) * u0.d[2],
                                  (va.x - v1.x) * u1.d[0] + (va.y - v1.y) * u1.d[1] + (va.z - v1.z) * u1.d[2]);
            }
        } else {
            const float4 x0 = P2[b0], x1 = P2[b1];
            float2 tb = make_float2(fmaxf(fmaf(q.r.x, -x0.w, 2.f), 0.f), fmaxf(fmaf(q.r.y, -x1.w, 2.f), 0.f));
            tb = __fmul2_rn(__fmul2_rn(tb, tb), tb);
            F = __fmul2_rn(__ffma2_rn(q.t3, both(cFa), make_float2(x0.y * tb.x, x1.y * tb.y)), both(0.5f));
        }
        acc.add_product(__fmul2_rn(m, vdr), F);
    };
    if (act) visit_list<G>(nbr, a, ld, ncnt[a], sub, body);
    const float sum = acc.template total<G>();
    float omt = om.x + om.y;
    if (VARH) {
#pragma unroll
        for (int o = 1; o < G; o <<= 1) omt += __shfl_xor_sync(0xffffffffu, omt, o);
    }
    if (!act || sub) return;
    float rate = sum;
    if (VARH) {
        const float hd1 = powi<ND>(iha) * iha;
        const float o = hd1 * (omt * wcon - va.w * ND * wK32(0.f, wcon));
        const float omega = 1.f + ha * o / (xa.x * ND);
        s.row(FD_OMEGA)[a] = omega;
        rate = EXPANDED ? sum / omega : sum * cFa / omega;
    }
    s.row(FD_DDDT)[a] += (double)rate;
}

/* Lanes per particle.  One lane runs the fewest instructions; more shorten
 * every lane's chain when the population leaves the chip short of warps.
 * Force pass, us with 1 / 4 / 8 lanes: 3D 3.8k 79 / 31 / 23, 23k 85 / 52 / 50,
 * 91k 135 / 114 / 141, 724k 530 / 684 / 978; 2D 6.5k 14.5 / 11.7 / 11.9, 23k
 * 13.4 / 17.3 / 22.  Continuity pass: 3D 3.8k 29 / 14 / 12, 23k 33 / 21 / 25,
 * 47k 36 / 37; 2D 6.5k 10.4 / 9.5, 23k 10.5 / 10.0.  (In 3D the force pass's
 * longest chains are those of the particles at a repulsive floor.  All in the
 * closed form: the coupled case's 8 lanes take the expanded one, 3.8k 26.7 and
 * 14.1 us, so that its continuity pass gains nothing over 4 lanes there.) */
int force_lanes(int64_t n, int nd) { return nd == 2 ? (n < 10000 ? 4 : 1) : (n < 12000 ? 8 : (n < 130000 ? 4 : 1)); }
int dddt_lanes(int64_t n, int nd) { return nd == 2 ? (n < 10000 ? 4 : 1) : (n < 12000 ? 8 : (n < 40000 ? 4 : 1)); }

}  // namespace

namespace mixed {

enum : int { CLASS_NONE = 0, CLASS_MORRIS, CLASS_MORRIS_VARH, CLASS_ARTIFICIAL };

static int force_class(const DevCfg &c) {
    if (c.nd == 1 || !(c.flags & SPHDEM_F_NO_ANTICLUMPING) || (c.flags & SPHDEM_F_CORRECTED_GRADIENT)) return CLASS_NONE;
    if (c.visc == SPHDEM_VISC_MORRIS) return c.var_h() ? CLASS_MORRIS_VARH : CLASS_MORRIS;
    if (c.visc == SPHDEM_VISC_ARTIFICIAL && !c.var_h()) return CLASS_ARTIFICIAL;
    return CLASS_NONE;
}

#define FORCE_CLASS_(M, ND, G, T)                                    \
    do {                                                             \
        if (cls == CLASS_MORRIS_VARH)                                \
            M(ND, SPHDEM_VISC_MORRIS, true, G, T);                   \
        else if (cls == CLASS_MORRIS)                                \
            M(ND, SPHDEM_VISC_MORRIS, false, G, T);                  \
        else                                                         \
            M(ND, SPHDEM_VISC_ARTIFICIAL, false, G, T);              \
    } while (0)
#define LANES_(M, ND, T)                \
    do {                                \
        if (lanes == 8)                 \
            M(ND, 8, T);                \
        else if (lanes == 4)            \
            M(ND, 4, T);                \
        else                            \
            M(ND, 1, T);                \
    } while (0)
#define TILES_(M, ND)                   \
    do {                                \
        if (tile)                       \
            LANES_(M, ND, true);        \
        else                            \
            LANES_(M, ND, false);       \
    } while (0)

bool force_lists(sphdem_ctx *c) {
    const int cls = force_class(c->cfg);
    if (cls == CLASS_NONE) return false;
    /* neighbour records staged through shared memory */
    const bool tile = c->force_tile;
    const size_t st_bytes = tile ? (size_t)3 * ST_CAP * sizeof(float4) : 0;
    const int lanes = force_lanes(c->n, c->cfg.nd);
#define LK_(ND, V, H, G, T)                                                                                       \
    SPHDEM_LAUNCH(c, "force32", (k_force_list<ND, V, H, G, T>), grid_for(c->n * G, c->blk_pair), c->blk_pair, st_bytes, \
                  c->cfg, c->dcfg, c->A, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_tg, c->mx_nbr,     \
                  c->mx_ncnt, (int64_t)c->mx_maxn, c->n, c->mx_nb, c->buf.start, c->buf.skey)
#define LG_(ND, G, T) FORCE_CLASS_(LK_, ND, G, T)
    if (c->cfg.nd == 3)
        TILES_(LG_, 3);
    else
        TILES_(LG_, 2);
#undef LG_
#undef LK_
    return true;
}

bool dddt_lists(sphdem_ctx *c) {
    if (c->cfg.nd == 1 || (c->cfg.flags & SPHDEM_F_CORRECTED_GRADIENT)) return false;
    const bool tile = c->force_tile;
    const size_t st_bytes = tile ? (size_t)2 * ST_CAP * sizeof(float4) : 0;
    const int lanes = dddt_lanes(c->n, c->cfg.nd);
#define LK_(ND, H, G, T)                                                                                          \
    SPHDEM_LAUNCH(c, "dddt32", (k_dddt_list<ND, H, G, T>), grid_for(c->n * G, c->blk_pair), c->blk_pair, st_bytes, \
                  c->cfg, c->A, c->g, c->mx_pos, c->mx_vel, c->mx_aux, c->mx_tg, c->mx_nbr, c->mx_ncnt,  \
                  (int64_t)c->mx_maxn, c->n, c->buf.start, c->buf.skey)
#define LG_(ND, G, T)              \
    do {                           \
        if (c->cfg.var_h())        \
            LK_(ND, true, G, T);   \
        else                       \
            LK_(ND, false, G, T);  \
    } while (0)
    if (c->cfg.nd == 3)
        TILES_(LG_, 3);
    else
        TILES_(LG_, 2);
#undef LG_
#undef LK_
    return true;
}

/* the dynamic shared memory of the staged forms */
void prepare_lists() {
    const int b3 = (int)(3 * ST_CAP * sizeof(float4)), b2 = (int)(2 * ST_CAP * sizeof(float4));
#define AF_(ND, V, H, G, T) \
    SPHDEM_CUDA_CHECK(cudaFuncSetAttribute(k_force_list<ND, V, H, G, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, b3))
#define AD_(ND, H, G, T) \
    SPHDEM_CUDA_CHECK(cudaFuncSetAttribute(k_dddt_list<ND, H, G, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, b2))
#define A_(ND, G)                                   \
    AF_(ND, SPHDEM_VISC_MORRIS, true, G, true);     \
    AF_(ND, SPHDEM_VISC_MORRIS, false, G, true);    \
    AF_(ND, SPHDEM_VISC_ARTIFICIAL, false, G, true); \
    AD_(ND, true, G, true);                         \
    AD_(ND, false, G, true)
    A_(2, 1);
    A_(2, 4);
    A_(2, 8);
    A_(3, 1);
    A_(3, 4);
    A_(3, 8);
#undef A_
#undef AD_
#undef AF_
}

}  // namespace mixed
}  // namespace sphdem
