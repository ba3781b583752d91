"""The work that programs built on this library have it do, as measurable cases.

Every case goes through the Python binding of the C ABI (``sphdem.capi``).  A
pass of the step cases is what a program does between two outputs: it gives
the handle the state it starts from, steps it, and reads the particles back
in tag order.  The adjoint cases are one gradient evaluation, the ensemble
case steps a batch, the hook case runs the phases one by one with a host hook
in between, as the case-directory driver does.

The inputs are the repository's own configurations (dam break, granular
settling, coupled sedimentation) in the middle of a run: particles off their
lattice and moving, spheres in contact.  Mixed-precision handles do their
pair sums in FP32, so what these sums give -- forces, velocities, densities,
gradients -- is taken as float32, and the FP64 positions as they are.

``exact`` restates one step (sphIncompress.cpp:3-251 and the functors it
runs) in plain torch float64, with gradients by autograd.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sph-dem_gb300"))
from sphdem import capi, cases  # noqa: E402

SPH, SPHB, BOUNDARY, DEM = cases.SPH, cases.SPH_BOUNDARY, cases.BOUNDARY, cases.DEM

# what a case leaves out takes these values
DEFAULTS = dict(kind="", prec="mixed", steps=10, n=1000, members=1, own=False, varh=True, ckpt=5)


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a first run or a unit test: about 1,400 particles, the plain FP64
        # path; the time is launches and latency
        dict(name="dambreak_tiny_fp64", kind="dambreak", prec="fp64", n=800, steps=20),
        # the 2D dam break at its full size, mixed and FP64
        dict(name="dambreak_mixed", kind="dambreak", prec="mixed", n=20000, steps=20),
        dict(name="dambreak_fp64", kind="dambreak", prec="fp64", n=20000, steps=10),
        # the damBreak case's own options: Monaghan viscosity, anticlumping,
        # h following density, corrected gradient, density re-initialisation
        # every step, adaptive dt
        dict(name="dambreak_own_options", kind="dambreak", prec="mixed", n=7001, steps=4, own=True),
        # granular settling at its full size: 50,000 polydisperse spheres,
        # half of them a bed in contact
        dict(name="dem_settling", kind="dem", prec="fp64", n=50000, steps=15),
        # coupled sedimentation, 3,800 particles: parameter studies, tests
        dict(name="sediment_small", kind="sediment", prec="mixed", n=3456, steps=10),
        # coupled sedimentation at its full size, the headline workload
        dict(name="sediment_full", kind="sediment", prec="mixed", n=1024000, steps=5),
        # the same physics in FP64 on a 1/16 box: validation runs
        dict(name="sediment_fp64", kind="sediment", prec="fp64", n=65536, steps=2),
        # an ensemble of dam breaks of many sizes in one batch
        dict(name="ensemble", kind="ensemble", prec="mixed", n=40000, members=16, steps=10),
        # a case directory's loop: phases one by one, a host hook that adds
        # the body force, output-step diagnostics at the end
        dict(name="hooks", kind="hooks", prec="mixed", n=21000, steps=3),
        # gradients of the coupled step (the 100k configuration) and of the
        # dam break, forward and backward
        dict(name="adjoint_sediment", kind="adjoint_sediment", prec="mixed", n=101306, steps=8, ckpt=4, varh=False),
        dict(name="adjoint_dambreak", kind="adjoint_dambreak", prec="fp64", n=20000, steps=16, ckpt=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dambreak", "dambreak", "dem", "sediment", "sediment", "ensemble", "hooks",
                       "adjoint_sediment", "adjoint_dambreak"])
    prec = rng.choice(["mixed", "fp64"])
    c = dict(kind=kind, prec=prec)
    if kind == "dambreak":
        c.update(n=_log_int(rng, 700, 120000), own=rng.random() < 0.3)
        c.update(steps=rng.randint(2, 5) if c["own"] else rng.randint(5, 20))
        if c["own"]:
            c["n"] = min(c["n"], 20011)
    elif kind == "dem":
        c.update(n=_log_int(rng, 1000, 120000), steps=rng.randint(5, 20))
    elif kind == "sediment":
        c.update(n=_log_int(rng, 3400, 700000 if prec == "mixed" else 40000),
                 steps=rng.randint(2, 5) if prec == "mixed" else 1, varh=rng.random() < 0.7)
    elif kind == "ensemble":
        c.update(n=_log_int(rng, 3000, 40000), members=rng.randint(3, 16), steps=rng.randint(3, 10), prec="mixed")
    elif kind == "hooks":
        c.update(n=_log_int(rng, 3400, 40000), steps=rng.randint(1, 3))
        if prec == "fp64":
            c["n"] = min(c["n"], 15001)
    elif kind == "adjoint_sediment":
        c.update(n=_log_int(rng, 3400, 90000), steps=rng.randint(3, 8), ckpt=rng.randint(2, 5), varh=rng.random() < 0.5,
                 prec="mixed")
    else:
        # few pairs under FP32: artificial viscosity has a kink at rest, and a pair that rounding
        # takes across it changes the gradient by more than rounding does
        small = prec == "mixed"
        c.update(n=_log_int(rng, 800, 2000 if small else 40000), steps=rng.randint(3, 5 if small else 20),
                 ckpt=rng.randint(2, 8))
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _rows(case):
    """Rows of the sediment lattice (nx x nx x 2 nx) for a fluid particle count."""
    return max(12, int(round((case["n"] / 2.0) ** (1.0 / 3.0))))


def _stir(p, sel, rng, dx, nd, speed, noise):
    """Particles off their lattice by up to 4 % of dx, in a smooth swirl plus noise."""
    m = int(sel.sum())
    r = p["r"]
    off = np.zeros((m, 3))
    off[:, :nd] = rng.uniform(-0.04 * dx, 0.04 * dx, (m, nd))
    r[sel] += off
    span = np.ptp(r[:, :nd], axis=0).max()
    k = 2 * math.pi / span
    ph = rng.uniform(0, 2 * math.pi, 3)
    x = r[sel]
    v = np.zeros((m, 3))
    for d in range(nd):
        v[:, d] = speed * np.sin(k * x[:, (d + 1) % nd] + ph[d])
    v[:, :nd] += noise * rng.standard_normal((m, nd))
    p["v"][sel] = v


def _dambreak(n, seed, own=False):
    rng = np.random.default_rng(seed)
    dx = math.sqrt(2.0 / n)
    kw = dict(visc_model=cases.VISC_MONAGHAN, anticlumping=True, const_h=False, viscosity=1e-2,
              corrected_gradient=True, reinit_every=1, fixed_dt=False) if own else {}
    c = cases.dambreak2d(dx=dx, seed=seed, jitter=0.01, **kw)
    cfg, p = c.cfg, c.particles
    fluid = p["iam"] == SPH
    # 10 % off the left wall, the side walls' layers untouched
    p["r"][fluid, 0] += 0.1 * dx
    _stir(p, fluid, rng, dx, 2, 0.5, 0.02)
    # hydrostatic density of the column, 2 m deep
    depth = np.clip(2.0 - p["r"][:, 1], 0.0, None)
    rho = 1000.0 * (1.0 + 7.0 * 1000.0 * 9.81 * depth / (1000.0 * cfg["spsound"] ** 2)) ** (1.0 / 7.0)
    p["dens"][fluid] = rho[fluid] * (1.0 + 1e-4 * rng.standard_normal(int(fluid.sum())))
    if own:
        p["h"][:] = 1.3 * (p["mass"] / p["dens"]) ** 0.5
    return cfg, p


def _dem(n, seed):
    rng = np.random.default_rng(seed)
    R, spread = 1e-3, 0.1
    nx = max(4, int(round((n / 20.0) ** 0.5)))
    nz = max(2, int(round(n / nx ** 2)))
    box = (2.0 * R * nx, 2.0 * R * nx, 6.0 * R * nz)
    c = cases.dem_settling3d(lattice=(nx, nx, nz), box=(box[0] * 1.4, box[1] * 1.4, 6.0 * R * nz), seed=seed)
    cfg, p = c.cfg, c.particles
    for d in range(2):
        cfg["rmax"][d] = box[d]
        cfg["walls"][2 * d + 1]["point"][d] = box[d]
    cfg["domain_min"], cfg["domain_max"] = [-0.25 * b for b in box], [1.25 * b for b in box]
    ii, jj, kk = np.meshgrid(np.arange(nx), np.arange(nx), np.arange(nz), indexing="ij")
    ii, jj, kk = ii.ravel(), jj.ravel(), kk.ravel()
    bed = nz // 2
    r = p["r"]
    r[:, 0], r[:, 1] = (ii + 0.5) * 2 * R, (jj + 0.5) * 2 * R
    # the lower half packed at one nominal diameter, the upper half falling
    r[:, 2] = np.where(kk < bed, (kk + 0.5) * 2 * R, 2 * R * bed + (kk - bed + 0.5) * 4 * R)
    r += rng.uniform(-0.02 * R, 0.02 * R, r.shape)
    p["v"][:] = 0.01 * rng.standard_normal(r.shape)
    p["v"][kk >= bed, 2] -= 0.3
    return cfg, p


def _sediment(nx, seed, varh=True, floor="boundary", dem_share=0.0488, viscosity=1e-6):
    """The coupled box at the full configuration's dx; L = nx dx, height 2 L."""
    rng = np.random.default_rng(seed)
    dx = 0.0025
    L, H = nx * dx, 2 * nx * dx
    c = cases.sediment3d(nx=nx, L=L, height=H, n_dem=1, seed=seed, floor=floor, var_h=varh, viscosity=viscosity)
    cfg, p = c.cfg, {k: v[:-1].copy() for k, v in c.particles.items()}   # the fluid and its floor
    R = c.notes["dem_radius"]
    vol = (4.0 / 3.0) * cases.REF_PI * R ** 3
    # spheres in the upper half: random cells of a lattice of 1.15 diameters, jittered inside
    w = 2.3 * R
    mx, mz = int(L / w), int((0.5 * H - 2 * R) / w)
    nd = max(20, min(int(dem_share * 2 * nx ** 3), (3 * mx * mx * mz) // 4))
    cell = rng.choice(mx * mx * mz, nd, replace=False)
    q = np.stack([cell // (mx * mz), (cell // mz) % mx, cell % mz], 1).astype(float)
    r = (q + 0.5) * np.array([L / mx, L / mx, w]) + rng.uniform(-0.15 * R, 0.15 * R, (nd, 3))
    r[:, 2] += 0.5 * H + R
    touching = rng.choice(nd // 2, max(1, nd // 10), replace=False) * 2   # a tenth in contact with the next one
    r[touching] = r[touching + 1] + 0.995 * 2 * R * np.eye(3)[rng.integers(0, 2, touching.size)]
    r[:, :2] %= L
    por = 1.0 - nd * vol / (L * L * 0.5 * H)
    cfg["coupling_radius"] = 1.999 * cfg["h"] / por ** (1.0 / 3.0)
    d = {k: np.zeros((nd,) + v.shape[1:], v.dtype) for k, v in p.items()}
    d["r"][:], d["iam"][:], d["radius"][:], d["h"][:] = r, DEM, R, R
    d["mass"][:], d["dens"][:], d["concave"][:] = vol * cfg["dem_dens"], cfg["dem_dens"], 1
    d["v"][:] = 0.01 * rng.standard_normal((nd, 3))
    d["v"][:, 2] -= 0.05
    fluid = p["iam"] == SPH
    _stir(p, fluid, rng, dx, 3, 0.02, 0.002)
    p["r"][fluid, :2] %= L
    # the pore pressure is near rest: rho = rho0 x local porosity, plus hydrostatics
    z = p["r"][:, 2]
    local = np.where((z > 0.5 * H) & (z < H - R), por, 1.0)
    head = np.clip(H - z, 0.0, None) * 9.81 / cfg["spsound"] ** 2
    p["dens"][fluid] = (1000.0 * local * (1.0 + head))[fluid] * (1.0 + 1e-4 * rng.standard_normal(int(fluid.sum())))
    if varh:
        own = (p["iam"] == SPH) | (p["iam"] == SPHB)
        p["h"][own] = 1.5 * np.cbrt(p["mass"][own] / p["dens"][own])
    p = {k: np.concatenate([p[k], d[k]]) for k in p}
    p["tag"] = np.arange(1, p["iam"].size + 1, dtype=np.int32)
    return cfg, p


def _inputs(case, seed):
    """[(cfg, particles)] of a case, one per member."""
    c = {**DEFAULTS, **case}
    k = c["kind"]
    if k in ("dambreak", "adjoint_dambreak"):
        return [_dambreak(c["n"], seed, c["own"])]
    if k == "dem":
        return [_dem(c["n"], seed)]
    if k == "ensemble":
        sizes = np.exp(np.linspace(math.log(2000), math.log(c["n"]), c["members"]))
        return [_dambreak(int(s), seed * 100 + i) for i, s in enumerate(sizes)]
    if k == "adjoint_sediment":
        return [_sediment(_rows(c), seed, c["varh"], floor="sphb3", viscosity=1e-5)]
    cfg, p = _sediment(_rows(c), seed, c["varh"])
    if k == "hooks":
        cfg["gravity_sph"] = [0.0, 0.0, 0.0]   # the host hook adds it
    return [(cfg, p)]


# --------------------------------------------------------------------------
# a pass
# --------------------------------------------------------------------------
_LIB = []
RESTART = ("r", "v", "vhat", "f", "fdrag", "dens", "h", "dddt")
RESTART_MASK = (capi.FIELD_R | capi.FIELD_V | capi.FIELD_VHAT | capi.FIELD_F | capi.FIELD_COUPLING | capi.FIELD_DENS
                | capi.FIELD_H | capi.FIELD_DDDT)
RESULT = ("r", "v", "f", "dens")
RESULT_MASK = capi.FIELD_R | capi.FIELD_V | capi.FIELD_F | capi.FIELD_DENS


class _Member:
    def __init__(self, lib, cfg, p, prec):
        n = p["iam"].size
        self.cfg, self.p, self.n, self.mixed = cfg, p, n, prec == "mixed"
        self.sim = capi.Simulation(lib, cfg, p, precision=cases.PREC_MIXED if self.mixed else cases.PREC_FP64)
        self.start = capi.ParticleBuffers(n, {k: p[k] for k in ("r", "v", "dens", "h")}, pinned=lib, fields=RESTART)
        self.out = capi.ParticleBuffers(n, pinned=lib, fields=RESULT)
        self.g0 = self.sim.globals()

    def rewind(self):
        self.sim.set(self.start, RESTART_MASK)
        self.sim.set_globals(self.g0)

    def result(self, fields=RESULT):
        self.sim.get(RESULT_MASK, self.out)
        return {k: _typed(self.out[k], self.mixed and k != "r") for k in fields}


def _typed(a, single):
    """The program's own copy of a field (the transfer buffers go with their handle)."""
    t = torch.from_numpy(a)
    return t.float() if single else t.clone()


def prepare(case, seed):
    c = {**DEFAULTS, **case}
    if not _LIB:
        _LIB.append(capi.Library())
    lib = _LIB[0]
    members = [_Member(lib, cfg, p, c["prec"]) for cfg, p in _inputs(case, seed)]
    st = dict(c, members=members)
    if c["kind"] == "ensemble":
        st["batch"] = capi.Batch(lib, [m.sim for m in members])
    if c["kind"] == "hooks":
        m = members[0]
        st["force"] = capi.ParticleBuffers(m.n, pinned=lib, fields=("f",))
        st["body"] = np.where((m.p["iam"] == SPH)[:, None], np.array([0.0, 0.0, -9.81]), 0.0)
    if c["kind"].startswith("adjoint"):
        m = members[0]
        m.sim.adjoint_set_tape_memory(-1)
        st["seeds"] = _seeds(m.p, seed)
    return st


def _seeds(p, seed):
    """dL/dr, dL/dv, dL/dvhat of the final state: a smooth weighting of the moving particles."""
    rng = np.random.default_rng(seed + 5)
    move = ((p["iam"] == SPH) | (p["iam"] == DEM))[:, None]
    return [np.where(move, rng.standard_normal((p["iam"].size, 3)) * s, 0.0) for s in (1.0, 0.1, 0.1)]


def run(st):
    kind, steps, m = st["kind"], st["steps"], st["members"][0]
    if kind == "ensemble":
        for q in st["members"]:
            q.rewind()
        st["batch"].step(steps)
        return [q.result(("r", "v", "dens")) for q in st["members"]]
    m.rewind()
    sim = m.sim
    if kind == "hooks":
        f = st["force"]
        for _ in range(steps):
            for ph in range(7):
                sim.phase(ph)
                if ph == capi.HOOK_BEFORE_MIDDLE:
                    sim.get(capi.FIELD_F, f)
                    f["f"][...] += st["body"]
                    sim.set(f, capi.FIELD_F)
        o = sim.output_vars()
        return {**m.result(), "e_ke": o["e_ke"], "max_v": o["max_v"], "ave_dens": o["ave_dens"]}
    if kind.startswith("adjoint"):
        sim.adjoint_forward(steps, st["ckpt"])
        out = m.result()
        g, dr, dv, dvh = sim.adjoint_backward(*st["seeds"])
        nd = m.cfg["ndim"]
        out.update({k: _typed(a[:, :nd].copy(), m.mixed) for k, a in (("dr0", dr), ("dv0", dv), ("dvhat0", dvh))})
        out["viscosity"] = g.viscosity
        if m.cfg["flags"] & cases.F_LIQ_DEM:
            out.update(drag_scale=g.drag_scale, dem_k=g.dem_k, dem_gamma=g.dem_gamma)
        return out
    sim.step(steps)
    return m.result()


def work(case):
    """Per step: the state (r, v, vhat, f, density, h, its rate, mass) read and written once; the pair
    terms of the force (60 operations) and of the continuity sum (30), both over each particle's
    neighbours, and of the two kernels' neighbour tests.  The adjoint is counted as two more steps."""
    c = {**DEFAULTS, **case}
    k = c["kind"]
    if k == "ensemble":
        sizes = np.exp(np.linspace(math.log(2000), math.log(c["n"]), c["members"]))
        n, nb, nd = float(1.25 * sizes.sum()), 20, 2
    elif k in ("dambreak", "adjoint_dambreak"):
        n, nb, nd = c["n"] + 22 * math.sqrt(c["n"] / 2.0), 20, 2
    elif k == "dem":
        n, nb, nd = c["n"], 6, 3
    else:
        nx = _rows(c)
        n, nb, nd = nx * nx * (2 * nx + 1) * 1.05, 113, 3
    passes = c["steps"] * (3 if k.startswith("adjoint") else 1)
    return {"bytes": passes * n * 2 * 8 * (4 * nd + 4), "flops": passes * n * nb * (90 + 2 * 10)}


# --------------------------------------------------------------------------
# the step in torch float64
# --------------------------------------------------------------------------
CHUNK = 12_000_000


def _near(ra, rb, reach, cfg):
    """Index pairs (i, j) and image shifts s with |ra_i - (rb_j + s)| <= reach."""
    nd, dev = cfg["ndim"], ra.device
    with torch.no_grad():
        lo = torch.tensor(cfg["domain_min"][:nd], device=dev, dtype=torch.float64)
        ext = torch.tensor(cfg["domain_max"][:nd], device=dev, dtype=torch.float64) - lo
        per = [bool(cfg["periodic"][d]) for d in range(nd)]
        num = [max(1, int(float(ext[d]) / (reach * 1.0000001))) for d in range(nd)]
        wid = ext / torch.tensor(num, device=dev, dtype=torch.float64)
        top = torch.tensor(num, device=dev) - 1

        def cell(r):
            return torch.minimum(torch.clamp(torch.floor((r[:, :nd] - lo) / wid).long(), min=0), top)

        def lin(c):
            k = c[:, 0]
            for d in range(1, nd):
                k = k * num[d] + c[:, d]
            return k

        kb = lin(cell(rb))
        order = torch.argsort(kb)
        cnt = torch.bincount(kb, minlength=int(math.prod(num)))
        first = torch.cumsum(cnt, 0) - cnt
        ca = cell(ra)
        I, J, S = [], [], []
        for o in np.ndindex(*(3,) * nd):
            t = ca + (torch.tensor(o, device=dev) - 1)
            ok = torch.ones(len(ra), dtype=torch.bool, device=dev)
            s = torch.zeros_like(ra[:, :nd])
            for d in range(nd):
                below, above = t[:, d] < 0, t[:, d] >= num[d]
                if per[d]:
                    s[:, d] = torch.where(below, -ext[d], torch.where(above, ext[d], s[:, d]))
                    t[:, d] = t[:, d] % num[d]
                else:
                    ok &= ~(below | above)
                    t[:, d] = t[:, d].clamp(0, num[d] - 1)
            k = lin(t)
            m = torch.where(ok, cnt[k], torch.zeros_like(k))
            i = torch.repeat_interleave(torch.arange(len(ra), device=dev), m)
            at = torch.arange(len(i), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
            j = order[first[k[i]] + at]
            d2 = ((ra[i, :nd] - rb[j, :nd] - s[i]) ** 2).sum(1)
            keep = d2 <= reach * reach
            i, j = i[keep], j[keep]
            I.append(i), J.append(j), S.append(s[i])
        return torch.cat(I), torch.cat(J), torch.cat(S)


def _chunks(pairs, whole):
    i, j, s = pairs
    size = max(1, len(i)) if whole else CHUNK
    for k in range(0, len(i), size):
        yield i[k:k + size], j[k:k + size], s[k:k + size]


def _K(q, wc):
    t = torch.clamp(2.0 - q, min=0.0)
    return wc * t ** 4 * (1.0 + 2.0 * q)


def _Fq(q, wc):
    """dK/dq / q of the Wendland C2 kernel."""
    return -10.0 * wc * torch.clamp(2.0 - q, min=0.0) ** 3


class _Model:
    """One configuration's step over a dict of float64 tensors, out of place."""

    def __init__(self, cfg, p, grad=False, hook_gravity=None):
        self.c, self.grad, self.hook = cfg, grad, hook_gravity
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.nd = nd = cfg["ndim"]
        iam = torch.as_tensor(p["iam"].astype(np.int64), device=dev)
        self.sph, self.bnd, self.dem = iam == SPH, iam == BOUNDARY, iam == DEM
        self.own = self.sph | (iam == SPHB)
        self.F = torch.nonzero(self.own | self.bnd)[:, 0]     # the fluid lists' particles
        self.O = torch.nonzero(self.own)[:, 0]
        self.D = torch.nonzero(self.dem)[:, 0]
        self.m, self.rad, self.n1 = t(p["mass"]), t(p["radius"]), t(p["norm1"])[:, :nd]
        self.n3 = t(p["norm3"])[:, :nd]
        self.wc = (7.0 / 64.0 if nd == 2 else 21.0 / 256.0) / cfg["pi"]
        fl = cfg["flags"]
        self.const_h, self.varh = bool(fl & cases.F_CONST_H), bool(fl & cases.F_VAR_H_CORRECTION)
        self.anti, self.cg = not fl & cases.F_NO_ANTICLUMPING, bool(fl & cases.F_CORRECTED_GRADIENT)
        self.liq, self.fixed = bool(fl & cases.F_LIQ_DEM), bool(fl & cases.F_FIXED_DT)
        z = torch.zeros_like(t(p["r"])[:, :nd])
        s = dict(r=t(p["r"])[:, :nd], v=t(p["v"])[:, :nd], vh=t(p["v"])[:, :nd], f=z, fp=z, fv=z, fb=z, fdrag=z,
                 dens=t(p["dens"]), h=t(p["h"]), dddt=torch.zeros_like(self.m), por=torch.ones_like(self.m))
        self.s, self.dt, self.time = s, cfg["maxdt"], 0.0
        self.par = {k: t(v) for k, v in dict(nu=cfg["viscosity"], alpha=cfg["alpha_artificial"], drag=cfg["drag_scale"],
                                             k=cfg["dem_k"], gam=cfg["dem_gamma"]).items()}

    def mask(self, sel, a, b):
        return torch.where(sel[:, None] if a.dim() > 1 else sel, a, b)

    def add(self, i, v, n=None):
        out = torch.zeros((len(self.m) if n is None else n,) + v.shape[1:], dtype=torch.float64, device=v.device)
        return out.index_add(0, i, v)

    def h_of(self, dens):
        return self.c["hfac"] * (self.m / dens) ** (1.0 / self.nd)

    def wrap(self, r):
        out = r.clone()
        for d in range(self.nd):
            if self.c["periodic"][d]:
                lo, hi = self.c["domain_min"][d], self.c["domain_max"][d]
                out[:, d] = r[:, d] + (hi - lo) * ((r[:, d] < lo).double() - (r[:, d] >= hi).double())
        return out

    def lists(self, r, h):
        """The fluid neighbour pairs: |r_a - r_b| <= 2 max(h_a, h_b), self left out."""
        i, j, s = _near(r[self.O].detach(), r[self.F].detach(), 2.0 * float(h[self.F].max()), self.c)
        i, j = self.O[i], self.F[j]
        keep = torch.cat([(i[k:k + CHUNK] != j[k:k + CHUNK])
                          & (((r[i[k:k + CHUNK]] - r[j[k:k + CHUNK]] - s[k:k + CHUNK]) ** 2).sum(1)
                             <= 4.0 * torch.maximum(h[i[k:k + CHUNK]], h[j[k:k + CHUNK]]) ** 2)
                          for k in range(0, max(1, len(i)), CHUNK)])
        return i[keep], j[keep], s[keep]

    def reinit(self, s):
        r, h = s["r"], self.mask(self.own, self.h_of(s["dens"]), s["h"])
        pairs = self.lists(r, h)
        i, j, sh = pairs
        keep = self.own[j]
        i, j, sh = i[keep], j[keep], sh[keep]
        d = torch.sqrt(((r[i] - r[j] - sh) ** 2).sum(1))
        dens = s["dens"]
        for k in range(10):
            if k:
                h = self.mask(self.own, self.h_of(dens), h)
            w = h ** -self.nd
            rho = self.m * w * _K(torch.zeros_like(h), self.wc) + self.add(i, self.m[j] * w[i] * _K(d / h[i], self.wc))
            dens = self.mask(self.own, rho, dens)
        return dict(s, dens=dens, h=h)

    def omega(self, r, h, dens, pairs):
        nd, ihn = self.nd, h ** -self.nd
        om = -self.m * nd * ihn / h * _K(torch.zeros_like(h), self.wc)
        for i, j, sh in _chunks(pairs, self.grad):
            q = torch.sqrt(((r[i] - r[j] - sh) ** 2).sum(1)) / h[i]
            term = self.m[j] * ihn[i] / h[i] * (-q * q * _Fq(q, self.wc) - nd * _K(q, self.wc))
            om = om + self.add(i, torch.where(self.own[j], term, torch.zeros_like(term)))
        return 1.0 + h * om / (dens * nd)

    def invm(self, r, h, dens, pairs):
        """calcInvM: M = -sum dvol gw (x) dx, gw the gradient with the sum's own removed."""
        i, j, sh = pairs
        nd = self.nd
        keep = self.own[j]
        i, j, sh = i[keep], j[keep], sh[keep]
        d = r[i] - r[j] - sh
        x = torch.sqrt((d ** 2).sum(1))
        hav = 0.5 * (h[i] + h[j])
        dvol = self.m[j] / dens[j]
        F = hav ** -(nd + 2) * _Fq(x / hav, self.wc)
        su = self.m / dens * h ** -nd * _K(torch.zeros_like(h), self.wc) + self.add(i, dvol * hav ** -nd * _K(x / hav, self.wc))
        cs = self.add(i, (dvol * F)[:, None] * d) / su[:, None]
        gw = (d * F[:, None] - cs[i]) / su[i][:, None]
        M = -self.add(i, dvol[:, None, None] * gw[:, :, None] * d[:, None, :])
        eye = torch.eye(nd, dtype=torch.float64, device=r.device)
        M = torch.where(self.own[:, None, None], M, eye)
        return torch.linalg.inv(M), cs, su

    def grads(self, cgs, i, d, F):
        if cgs is None:
            return d * F[:, None]
        M, cs, su = cgs
        return torch.einsum("pij,pj->pi", M[i], (d * F[:, None] - cs[i]) / su[i][:, None])

    def force(self, s, pairs, om, cgs, pdr2):
        c, nd, wc = self.c, self.nd, self.wc
        r, vh, h, dens, m = s["r"], s["vh"], s["h"], s["dens"], self.m
        fp, fv, fb, fa = (torch.zeros_like(r) for _ in range(4))
        ndt = [float("inf")]
        k_anti = wc * (2.0 - 1.0 / c["hfac"]) ** 4 * (1.0 + 2.0 / c["hfac"])
        for i, j, sh in _chunks(pairs, self.grad):
            d = r[i] - r[j] - sh
            r2 = (d ** 2).sum(1)
            x = torch.sqrt(r2)
            Fa, Fb = h[i] ** -(nd + 2) * _Fq(x / h[i], wc), h[j] ** -(nd + 2) * _Fq(x / h[j], wc)
            ga, gb = self.grads(cgs, i, d, Fa), self.grads(cgs, i, d, Fb)
            if self.varh:
                ga, gb = ga / om[i][:, None], gb / om[i][:, None]
            else:
                ga = gb = 0.5 * (ga + gb)
            gm = 0.5 * (ga + gb)
            dv, hav = vh[i] - vh[j], 0.5 * (h[i] + h[j])
            vdr = (d * dv).sum(1)
            isph = self.sph[i]
            one = torch.ones_like(x)
            if c["visc_model"] == cases.VISC_MORRIS:
                num = 2.0 * self.par["nu"] * c["dens"] if self.liq else self.par["nu"] * (dens[i] + dens[j])
                fvp = dv * (m[j] * num / (dens[i] * dens[j]) * (d * gm).sum(1) / (r2 + 0.01 * hav ** 2))[:, None]
                vsig, to = 2.0 * c["spsound"] * one, "v"
            elif c["visc_model"] == cases.VISC_MONAGHAN:
                vs = vdr / x
                vsig, to = 2.0 * c["spsound"] + 2.0 * vs.abs(), "v"
                al = self.par["nu"] * (112.0 / 15.0) / (c["spsound"] * c["h"])
                fvp = gm * (m[j] * vs * vsig * al / (dens[i] + dens[j]))[:, None]
            else:
                vs = torch.where(vdr < 0, vdr / x, torch.zeros_like(x))
                vsig, to = 2.0 * c["spsound"] - 4.0 * vs, "a"
                fvp = gm * (m[j] * vs * vsig * self.par["alpha"] / (dens[i] + dens[j]))[:, None]
            fvp = torch.where(isph[:, None], fvp, torch.zeros_like(fvp))
            fv, fa = (fv + self.add(i, fvp), fa) if to == "v" else (fv, fa + self.add(i, fvp))
            if not self.fixed and bool(isph.any()):
                vdc = 0.06 if c["visc_model"] == cases.VISC_MONAGHAN else 0.125
                ndt += [float((0.6 * hav / vsig)[isph].min()), float((vdc * hav ** 2 / c["viscosity"])[isph].min())]
            anti = 0.01 * (pdr2[i] + pdr2[j]).abs() * (_K(x / hav, wc) / k_anti) ** 4 if self.anti else 0.0 * x
            fpp = -m[j][:, None] * (pdr2[i][:, None] * ga + pdr2[j][:, None] * gb + anti[:, None])
            b = self.bnd[j]
            fp = fp + self.add(i, torch.where(b[:, None], torch.zeros_like(fpp), fpp))
            if bool(b.any()):
                fb = fb + self.add(i[b], self.wall_particle(i[b], j[b], d[b], dv[b]))
        return fp, fv, fb, fa, min(ndt)

    def wall_particle(self, i, j, d, dv):
        """Repulsive boundary particles of a flat floor (one normal)."""
        c, n = self.c, self.n1[j]
        perp = (n * d).sum(1)
        rt = d - perp[:, None] * n
        pt0 = (rt * self.n3[j]).sum(1).abs()
        pt1 = torch.sqrt((torch.linalg.cross(rt, self.n3[j]) ** 2).sum(1))
        dp = 1.0 / (c["bfac"] * c["psep"])
        pesky = 0.25 * (1 + torch.cos(c["pi"] * pt0 * dp)) * (1 + torch.cos(c["pi"] * pt1 * dp))
        q = perp.abs() / c["psep"]
        c0 = c["spsound"]
        big = 0.01 * c0 * c0 - torch.where((d * dv).sum(1) < 0, 1.0, 0.0) * c0 * (dv * n).sum(1)
        law = torch.where(q <= 2.0 / 3.0, torch.full_like(q, 2.0 / 3.0),
                          torch.where(q <= 1.0, 2.0 * q - 1.5 * q * q, 0.5 * (2.0 - q) ** 2)) / perp.abs()
        mag = torch.sign(perp) * 2.0 * self.m[i] / (self.m[i] + self.m[j]) * big * law * pesky
        on = (pt0 * dp <= 1.0) & (pt1 * dp <= 1.0) & (q < 2.0)
        return torch.where(on[:, None], mag[:, None] * n, torch.zeros_like(n))

    def coupled(self, r):
        """Fluid -> sphere pairs by the reference's bucket rule (dataLL.cpp:1154-1190)."""
        c, nd = self.c, self.nd
        i, j, s = _near(r[self.O].detach(), r[self.D].detach(), c["coupling_radius"], c)
        i, j = self.O[i], self.D[j]
        rc, sr = c["coupling_radius"], c["dem_search_radius"]
        num, lim = math.ceil(0.5 * rc / sr), (0.5 * rc / sr) ** 2
        lo = torch.tensor(c["domain_min"][:nd], device=r.device, dtype=torch.float64)
        bucket = lambda x: torch.trunc((x - lo) / (2 * sr) + (2 * rc / sr - 1)).long()  # noqa: E731
        o = bucket((r[j] + s).detach()) - bucket(r[i].detach())
        ok = (o.abs() <= num).all(1) & ((((o + 1) ** 2).sum(1) < lim) | (((o - 1) ** 2).sum(1) < lim))
        return i[ok], j[ok], s[ok]

    def middle_coupling(self, s):
        c, nd, wc = self.c, self.nd, self.wc
        r, hc = s["r"], c["coupling_radius"] / 2.0
        pairs = self.coupled(r)
        dvol = self.m / s["dens"]
        por, shep = torch.zeros_like(self.m), torch.zeros_like(self.m)
        inc = (4.0 / 3.0) * c["pi"] * c["dem_radius"] ** 3
        for i, j, sh in _chunks(pairs, self.grad):
            W = hc ** -nd * _K(torch.sqrt(((r[i] - r[j] - sh) ** 2).sum(1)) / hc, wc)
            por, shep = por + self.add(i, inc * W), shep + self.add(j, dvol[i] * W)
        fd = torch.zeros_like(r)
        for i, j, sh in _chunks(pairs, self.grad):
            W = hc ** -nd * _K(torch.sqrt(((r[i] - r[j] - sh) ** 2).sum(1)) / hc, wc)
            fd = fd - self.add(i, s["fdrag"][j] * (self.m[j] / s["dens"][i] * W / shep[j])[:, None])
        por = torch.clamp(1.0 - por, min=0.37)
        return self.mask(self.own, por, torch.ones_like(por)), self.mask(self.own, fd, s["fdrag"])

    def end_spheres(self, s):
        """calcFPI, Di Felice drag and the contacts; s already holds the walls and gravity."""
        c, nd, wc, D = self.c, self.nd, self.wc, self.D
        r, vh, h, m = s["r"], s["vh"], s["h"], self.m
        f, fp, fdrag = s["f"], s["fp"], s["fdrag"]
        if len(self.O):
            reach = 2.0 * max(float(h[self.O].max()), float(h[D].max()))
            i, j, sh = _near(r[D].detach(), r[self.O].detach(), reach, c)
            i, j = D[i], self.O[j]
            d = torch.sqrt(((r[i] - r[j] - sh) ** 2).sum(1))
            keep = d <= 2.0 * torch.maximum(h[i], h[j])
            i, j, d = i[keep], j[keep], d[keep]
            W = h[j] ** -nd * _K(d / h[j], wc)
            dvw = m[j] / s["dens"][j] * W
            total = self.add(i, dvw)
            fpfb = self.add(i, (m[j] * W)[:, None] * (s["fp"][j] + s["fb"][j]))
            fv = self.add(i, (m[j] * W + dvw)[:, None] * s["fv"][j])
            vel, por = self.add(i, dvw[:, None] * vh[j]), self.add(i, dvw * s["por"][j])
            on = self.dem & (total > 0.5)
            safe = torch.where(on, total, torch.ones_like(total))
            fpfb, fv, vel, por = fpfb / safe[:, None], fv / safe[:, None], vel / safe[:, None], por / safe
            dv = por[:, None] * (vel - vh)
            v2 = (dv ** 2).sum(1)
            speed = torch.sqrt(torch.where(on, v2, torch.ones_like(v2)))
            por_s = torch.where(on, por, torch.ones_like(por))
            Re = 2.0 * c["dem_radius"] / self.par["nu"] * speed
            power = 3.7 - 0.65 * torch.exp(-(1.5 - torch.log10(Re)) ** 2 / 2.0)
            mag = 0.5 * c["pi"] * c["dem_radius"] ** 2 * (0.63 + 4.8 / torch.sqrt(Re)) ** 2 * speed * por_s ** -power
            drag = (c["dem_vol"] / m)[:, None] * (fv + fpfb) + (c["dens"] / m * self.par["drag"] * mag)[:, None] * dv
            drag = torch.where(on[:, None], drag, torch.zeros_like(drag))
            fdrag = self.mask(self.dem, drag, fdrag)
            f = f + drag
        i, j, sh = _near(r[D].detach(), r[D].detach(), 2.0 * float(h[D].max()), c)
        i, j, sh = D[i], D[j], sh
        d = r[i] - r[j] - sh
        x2 = (d ** 2).sum(1)
        keep = (i != j) & (x2 <= 4.0 * torch.maximum(h[i], h[j]) ** 2)
        i, j, d, x = i[keep], j[keep], d[keep], torch.sqrt(x2[keep])
        ra = torch.where(self.rad > 0, self.rad, torch.full_like(self.rad, c["dem_radius"]))
        lap = ra[i] + ra[j] - x
        keep = lap > 0
        i, j, nrm, lap = i[keep], j[keep], d[keep] / x[keep][:, None], lap[keep]
        mag = self.par["k"] * lap - self.par["gam"] * ((vh[i] - vh[j]) * nrm).sum(1)
        fc = self.add(i, nrm * (mag / m[i])[:, None])
        return f + fc, fp + fc, fdrag

    def step(self, s):
        c, nd, dt = self.c, self.nd, self.dt
        hd = 0.5 * dt
        sph, own, dem = self.sph, self.own, self.dem
        z = torch.zeros_like(s["r"])
        s = dict(s)
        v0, vh0 = s["v"], s["vh"]
        s["r"] = self.wrap(s["r"] + hd * self.mask(own | dem, s["vh"], z))
        s["vh"], s["v"] = self.mask(sph, s["vh"] + hd * s["f"], s["vh"]), self.mask(sph, s["v"] + hd * s["f"], s["v"])
        s["dens"] = self.mask(own, s["dens"] + hd * s["dddt"], s["dens"])
        if not self.const_h:
            s["h"] = self.mask(own, self.h_of(s["dens"]), s["h"])
        for k in ("f", "fp", "fv", "fb"):
            s[k] = self.mask(own, z, s[k])
        if c["reinit_dens_every"]:
            s = self.reinit(s)
        g = torch.tensor(self.hook or c["gravity_sph"][:nd], dtype=torch.float64, device=z.device)
        s["f"] = self.mask(sph, s["f"] + g, s["f"])
        ndt = c["maxdt"]
        if len(self.O):
            if self.liq:
                s["por"], s["fdrag"] = self.middle_coupling(s)
                s["f"] = self.mask(own, s["f"] + s["fdrag"], s["f"])
            pairs = self.lists(s["r"], s["h"].detach())
            om = self.omega(s["r"], s["h"], s["dens"], pairs) if self.varh else None
            cgs = self.invm(s["r"], s["h"], s["dens"], pairs) if self.cg else None
            x = s["dens"] / (c["refd"] * s["por"])
            pdr2 = c["prb"] * (x ** 7 - 1.0) / s["dens"] ** 2
            fp, fv, fb, fa, lim = self.force(s, pairs, om, cgs, pdr2)
            s["fp"], s["fv"], s["fb"] = s["fp"] + fp, s["fv"] + fv, s["fb"] + fb
            s["f"] = s["f"] + fp + fv + fb + fa
            ndt = min(ndt, lim)
            if not self.fixed:
                acc = 0.25 * torch.sqrt(s["h"] / torch.sqrt((s["f"] ** 2).sum(1)))
                ndt = min(ndt, float(acc[own].min()))
            del pairs
        new = dt if self.fixed else ndt
        kick = 0.5 * dt + 0.5 * new
        old_hd, self.dt = hd, new
        dt, hd = new, 0.5 * new
        s["v"], s["vh"] = self.mask(sph, v0 + kick * s["f"], s["v"]), self.mask(sph, vh0 + kick * s["f"], s["vh"])
        if len(self.D):
            s["r"] = s["r"] + hd * self.mask(dem, s["vh"], z)
            s["v"], s["vh"] = self.mask(dem, s["v"] + hd * s["f"], s["v"]), self.mask(dem, s["vh"] + hd * s["f"], s["vh"])
            s["f"] = self.mask(dem, torch.tensor(c["gravity_dem"][:nd], dtype=torch.float64, device=z.device) + z, s["f"])
            for k in ("fp", "fv", "fb"):
                s[k] = self.mask(dem, z, s[k])
            ra = torch.where(self.rad > 0, self.rad, torch.full_like(self.rad, c["dem_radius"]))
            for w in c["walls"]:
                n = torch.tensor(w["normal"], dtype=torch.float64, device=z.device)
                pt = torch.tensor([float(x) for x in w["point"]], dtype=torch.float64, device=z.device)
                lap = ra - ((s["r"] - pt) * n).sum(1)
                mag = (self.par["k"] * lap - self.par["gam"] * (s["vh"] * n).sum(1)) / self.m
                fw = torch.where((dem & (lap > 0))[:, None], mag[:, None] * n, z)
                s["f"] = s["f"] + fw
        s["r"] = self.wrap(s["r"] + hd * self.mask(own, s["vh"], z))
        if len(self.O):
            pairs = self.lists(s["r"], s["h"].detach())
            om = self.omega(s["r"], s["h"], s["dens"], pairs) if self.varh else None
            cgs = self.invm(s["r"], s["h"], s["dens"], pairs) if self.cg else None
            rate = torch.zeros_like(self.m)
            for i, j, sh in _chunks(pairs, self.grad):
                d = s["r"][i] - s["r"][j] - sh
                x = torch.sqrt((d ** 2).sum(1))
                w = self.grads(cgs, i, d, s["h"][i] ** -(nd + 2) * _Fq(x / s["h"][i], self.wc))
                if self.varh:
                    w = w / om[i][:, None]
                else:
                    w = 0.5 * (w + self.grads(cgs, i, d, s["h"][j] ** -(nd + 2) * _Fq(x / s["h"][j], self.wc)))
                term = self.m[j] * ((s["vh"][i] - s["vh"][j]) * w).sum(1)
                rate = rate + self.add(i, torch.where(self.own[j], term, torch.zeros_like(term)))
            s["dddt"] = self.mask(own, rate, s["dddt"])
        if len(self.D):
            s["f"], s["fp"], s["fdrag"] = self.end_spheres(s)
            v_mid, vh_mid = v0, vh0
            s["v"], s["vh"] = self.mask(dem, v_mid + dt * s["f"], s["v"]), self.mask(dem, vh_mid + dt * s["f"], s["vh"])
        if len(self.O):
            s["dens"] = self.mask(own, s["dens"] + hd * s["dddt"], s["dens"])
            if not self.const_h:
                s["h"] = self.mask(own, self.h_of(s["dens"]), s["h"])
        return s


def _result(model, s, keys=RESULT):
    pad = lambda a: torch.nn.functional.pad(a, (0, 3 - a.shape[1])) if a.dim() > 1 else a  # noqa: E731
    return {k: pad(s[k].detach()) for k in keys}


def exact(case, seed):
    c = {**DEFAULTS, **case}
    if c["kind"].startswith("adjoint"):
        return _exact_adjoint(c, seed, *_inputs(case, seed)[0])
    outs = []
    for cfg, p in _inputs(case, seed):
        with torch.no_grad():
            m = _Model(cfg, p, hook_gravity=[0.0, 0.0, -9.81] if c["kind"] == "hooks" else None)
            s = m.s
            for _ in range(c["steps"]):
                s = m.step(s)
        o = _result(m, s, ("r", "v", "dens") if c["kind"] == "ensemble" else RESULT)
        if c["kind"] == "hooks":
            o["e_ke"] = float((0.5 * m.m * (s["vh"] ** 2).sum(1))[m.sph].sum())
            o["max_v"] = float(torch.sqrt((s["v"] ** 2).sum(1))[m.own].max())
            o["ave_dens"] = float(s["dens"][m.own].sum()) / len(m.m)
        outs.append(o)
    return outs if c["kind"] == "ensemble" else outs[0]


def _exact_adjoint(c, seed, cfg, p):
    from torch.utils.checkpoint import checkpoint
    m = _Model(cfg, p, grad=True)
    keys = list(m.s)
    lead = {k: m.s[k].clone().requires_grad_(True) for k in ("r", "v", "vh")}
    par = {k: v.requires_grad_(True) for k, v in m.par.items()}

    def one(*flat):
        return tuple(m.step(dict(zip(keys, flat)))[k] for k in keys)

    flat = tuple({**m.s, **lead}[k] for k in keys)
    for _ in range(c["steps"]):
        flat = checkpoint(one, *flat, use_reentrant=False)
    s = dict(zip(keys, flat))
    nd = cfg["ndim"]
    w = [torch.as_tensor(a[:, :nd].copy(), device=s["r"].device) for a in _seeds(p, seed)]
    loss = (w[0] * s["r"]).sum() + (w[1] * s["v"]).sum() + (w[2] * s["vh"]).sum()
    liq = bool(cfg["flags"] & cases.F_LIQ_DEM)
    names = ["nu", "drag", "k", "gam"] if liq else ["alpha"]
    g = torch.autograd.grad(loss, [lead["r"], lead["v"], lead["vh"]] + [par[k] for k in names], allow_unused=True)
    out = _result(m, s)
    out.update(dr0=g[0], dv0=g[1], dvhat0=g[2])
    for k, v in zip(["viscosity", "drag_scale", "dem_k", "dem_gamma"], g[3:]):
        out[k] = 0.0 if v is None else float(v)
    return out
