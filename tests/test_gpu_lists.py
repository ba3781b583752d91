"""Neighbour lists of the mixed path on awkward populations (-m gpu): counts
around the warp's 32 particles and around the point where the build changes
from four lanes per particle to one, random clouds with unequal h, exact ties
(a lattice with neighbours at exactly 2h) and periodic images.  The lists must
hold exactly the pairs of the FP64 bucket scan."""
import copy

import numpy as np
import pytest

from sphdem import capi, cases
from sphdem.state import pair_set

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__
    __graft_entry__.build()
    return capi.Library()


def cloud(nd, n, tie, seed=5):
    """n sph particles in a box of the density of the named workload."""
    rng = np.random.default_rng(seed)
    base = cases.workload("dambreak2d_small" if nd == 2 else "sediment3d_small")
    cfg = copy.deepcopy(base.cfg)
    dx = cfg["psep"]
    side = int(np.ceil(n ** (1.0 / nd)))
    ext = max(side * dx, 10 * dx)
    cfg["rmin"], cfg["rmax"] = [0.0] * 3, [ext] * nd + [0.0] * (3 - nd)
    cfg["domain_min"] = [0.0 if cfg["periodic"][d] else -4 * dx for d in range(nd)] + [0.0] * (3 - nd)
    cfg["domain_max"] = [ext if cfg["periodic"][d] else ext + 4 * dx for d in range(nd)] + [0.0] * (3 - nd)
    p = cases._empty_particles(n)
    q = np.stack(np.unravel_index(rng.permutation(side ** nd)[:n], (side,) * nd), 1) + 0.5
    p["r"][:, :nd] = q * dx if tie else rng.uniform(0.0, ext, (n, nd))
    p["mass"][:], p["dens"][:] = dx ** nd * 1000.0, 1000.0
    p["h"][:] = 1.5 * dx if tie else 1.3 * dx * rng.uniform(0.8, 1.1, n)
    return cfg, p


@pytest.mark.parametrize("nd,n", [(2, 1), (2, 31), (2, 33), (2, 300), (2, 64990), (2, 65010),
                                  (3, 32), (3, 129), (3, 1000), (3, 39990), (3, 40010)])
@pytest.mark.parametrize("tie", [False, True])
def test_lists_equal_the_fp64_bucket_scan(lib, nd, n, tie):
    cfg, p = cloud(nd, n, tie)
    sets = []
    for prec in (cases.PREC_FP64, cases.PREC_MIXED):
        sim = capi.Simulation(lib, cfg, p, precision=prec)
        sets.append(pair_set(*sim.pairs(capi.PAIRS_SPH)))
        sim.close()
    assert n < 30 or sets[0].size > 0
    assert np.array_equal(sets[0], sets[1])


def list_pass_case(kind, n):
    """Moving, slightly disordered fluid with walls; `n` sets the lanes per particle."""
    rng = np.random.default_rng(3)
    if kind == "artificial":
        case = cases.dambreak2d(dx=float(np.sqrt(2.0 / n)))
    else:
        nx = int(round((n / 2.0) ** (1.0 / 3.0)))
        case = cases.sediment3d(nx=nx, L=0.0025 * nx, height=0.005 * nx, n_dem=20, viscosity=1e-4,
                                var_h=kind == "morris_varh")
    p, nd, dx = case.particles, case.cfg["ndim"], case.cfg["psep"]
    fluid = p["iam"] == cases.SPH
    p["r"][fluid, :nd] += rng.uniform(-0.05 * dx, 0.05 * dx, (int(fluid.sum()), nd))
    p["v"][fluid, :nd] += 0.05 * rng.standard_normal((int(fluid.sum()), nd))
    for d in range(nd):
        if case.cfg["periodic"][d]:
            p["r"][fluid, d] %= case.cfg["rmax"][d]
    p["dens"][fluid] *= 1.0 + 1e-3 * rng.standard_normal(int(fluid.sum()))
    return case, fluid


@pytest.mark.parametrize("kind", ["artificial", "morris", "morris_varh"])
@pytest.mark.parametrize("n", [1800, 7000, 16000, 132000])
def test_list_passes_equal_fp64(lib, kind, n):
    """Force and continuity passes, one to eight lanes per particle: pressure,
    viscous and wall forces, density rate and Omega against the FP64 path.
    Tolerance: FP32 terms good to ~20 roundings (1.2e-6) of which a sum
    cancels at most nine tenths (2-norm over the fluid)."""
    case, fluid = list_pass_case(kind, n)
    got = []
    for prec in (cases.PREC_FP64, cases.PREC_MIXED):
        sim = capi.Simulation(lib, case.cfg, case.particles, precision=prec)
        sim.step(1)
        a = sim.get()
        got.append({k: a[k][fluid].copy() for k in ("f", "fp", "fv", "fb", "dddt", "omega")})
        sim.close()
    for k, x in got[0].items():
        norm = np.linalg.norm(x)
        if norm > 0:
            assert np.linalg.norm(got[1][k] - x) <= 1.2e-5 * norm, k


@pytest.mark.parametrize("kind,n", [("artificial", 1800), ("options", 1800)])
def test_fp64_particles_beyond_the_list_depth(lib, kind, n):
    """An FP64 handle squeezed beyond the depth its lists were given at
    creation scans the buckets instead: the step equals that of a handle
    created at the squeezed positions (whose lists are deep enough), up to
    the order of the FP64 sums (1e-12 of each field's 2-norm)."""
    if kind == "options":
        case = cases.dambreak2d(dx=0.05, visc_model=cases.VISC_MONAGHAN, anticlumping=True, const_h=False, var_h=True,
                                viscosity=1e-2, reinit_every=1, fixed_dt=False)
        fluid = case.particles["iam"] == cases.SPH
    else:
        case, fluid = list_pass_case(kind, n)
    nd = case.cfg["ndim"]
    r = case.particles["r"].copy()
    mid = r[fluid].mean(axis=0)
    r[fluid, nd - 1] = mid[nd - 1] + 0.3 * (r[fluid, nd - 1] - mid[nd - 1])
    r[fluid, 0] = mid[0] + 0.5 * (r[fluid, 0] - mid[0])
    got = []
    for squeezed in (False, True):
        p = dict(case.particles, r=r) if squeezed else case.particles
        sim = capi.Simulation(lib, case.cfg, p, precision=cases.PREC_FP64)
        buf = capi.ParticleBuffers(case.n, {"r": r}, fields=("r",))
        sim.set(buf, capi.FIELD_R)
        sim.rebuild()
        sim.rebuild()   # the ghost widths of both handles follow the same h
        sim.step(1)
        a = sim.get()
        got.append({k: a[k][fluid].copy() for k in ("f", "fp", "dddt", "dens")})
        sim.close()
    for k in got[0]:
        assert np.linalg.norm(got[0][k] - got[1][k]) <= 1e-12 * np.linalg.norm(got[1][k]), k
