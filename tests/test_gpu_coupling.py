"""Coupling and contact passes at the edges of their queues and splits (-m
gpu): more partners per fluid particle than a queue or the kept pairs hold,
populations on both sides of the four-threads rule, contacts beyond a lane's
queue, DEM without fluid.  Checked against the CPU oracle (FP64, 1e-11 of each
field's 2-norm: sums of some hundred terms in another order) and, for mixed
precision, against the FP64 path (FP32 terms of ~20 roundings, 1.2e-5)."""
import numpy as np
import pytest

from oracle.port_api import OracleSim
from sphdem import capi, cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__
    __graft_entry__.build()
    return capi.Library()


def dense_bed(nx, spacing, seed=4):
    """A sediment box whose upper half holds spheres `spacing` diameters apart
    on a jittered lattice (spacing < 1: every sphere in contact)."""
    case = cases.sediment3d(nx=nx, L=0.0025 * nx, height=0.005 * nx, n_dem=1)
    p, cfg = case.particles, case.cfg
    R, L = cfg["dem_radius"], cfg["rmax"][0]
    m = int(L / (2 * R * spacing))
    k = max(2, int((0.5 * cfg["rmax"][2] - 4 * R) / (2 * R * spacing)))
    rng = np.random.default_rng(seed)
    q = np.stack(np.meshgrid(np.arange(m), np.arange(m), np.arange(k), indexing="ij"), -1).reshape(-1, 3)
    r = (q + 0.5) * np.array([L / m, L / m, 2 * R * spacing]) + rng.uniform(-0.02 * R, 0.02 * R, q.shape)
    r[:, 2] += 0.5 * cfg["rmax"][2] + R
    r[:, :2] %= L
    n = len(r)
    out = {key: np.concatenate([v[:-1], np.repeat(v[-1:], n, axis=0)]) for key, v in p.items()}
    out["r"][-n:] = r
    out["v"][-n:] = 0.02 * rng.standard_normal((n, 3))
    out["tag"] = np.arange(1, out["iam"].size + 1, dtype=np.int32)
    # the pore pressure at rest: the spheres take a good part of the volume
    fluid = (out["iam"] == cases.SPH) & (out["r"][:, 2] > 0.5 * cfg["rmax"][2])
    out["dens"][fluid] *= 1.0 - n * cfg["dem_vol"] / (L * L * 0.5 * cfg["rmax"][2])
    return cfg, out


FIELDS = ("f", "fp", "fdrag", "fvel", "porosity", "dporositydt", "grad_porosity", "shep_sum", "dddt")


def norm_gap(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / n if n > 0 else np.linalg.norm(a)


@pytest.mark.parametrize("spacing", [0.98, 1.3, 2.5])
def test_dense_suspension_equals_oracle(lib, spacing):
    cfg, p = dense_bed(12, spacing)
    ora = OracleSim(cfg, p)
    ora.step(1)
    want = ora.get()
    sim = capi.Simulation(lib, cfg, p, precision=cases.PREC_FP64)
    sim.step(1)
    got = sim.get()
    for k in FIELDS:
        assert norm_gap(got[k], want[k]) <= 1e-11, k


@pytest.mark.parametrize("nx,spacing", [(12, 0.98), (30, 1.1), (32, 1.1)])
def test_mixed_coupling_equals_fp64(lib, nx, spacing):
    cfg, p = dense_bed(nx, spacing)
    got = []
    for prec in (cases.PREC_FP64, cases.PREC_MIXED):
        sim = capi.Simulation(lib, cfg, p, precision=prec)
        sim.step(1)
        a = sim.get()
        got.append({k: a[k].copy() for k in FIELDS})
        sim.close()
    for k in FIELDS:
        assert norm_gap(got[1][k], got[0][k]) <= 1.2e-5, k


@pytest.mark.parametrize("precision", [cases.PREC_FP64, cases.PREC_MIXED])
def test_crowded_contacts_without_fluid(lib, precision):
    """Spheres squeezed to half a diameter: more contacts per lane than its
    queue holds (FP64 on both handles)."""
    case = cases.dem_settling3d(lattice=(6, 6, 10), box=(0.0138, 0.0138, 0.023), spread=0.0, vel_amp=0.1)
    p = case.particles
    p["r"][:] = p["r"].mean(axis=0) + 0.45 * (p["r"] - p["r"].mean(axis=0))
    ora = OracleSim(case.cfg, p)
    ora.step(1)
    want = ora.get()
    sim = capi.Simulation(lib, case.cfg, p, precision=precision)
    sim.step(1)
    got = sim.get()
    for k in ("f", "fp", "v", "r", "fdrag", "shep_sum"):
        assert norm_gap(got[k], want[k]) <= 1e-11, k


@pytest.mark.parametrize("nx", [12, 32])
def test_fluid_inserted_into_a_handle_of_dem_only(lib, nx):
    """A mixed handle of DEM only runs the FP64 passes, also once fluid has been
    inserted up to its capacity, with more partners per fluid particle than the
    kept pairs hold (four threads a particle, and one): the step of an FP64
    handle created with all particles.  Both sum in FP64; the mixed handle takes
    h and the reciprocals of the equation of state by a Newton step good to
    1e-14, which the pressure (x^7 - 1) and its differences enlarge by up to
    some 1e4: 1e-9 of each field's 2-norm."""
    cfg, p = dense_bed(nx, 0.98)
    order = np.argsort(p["iam"] != cases.DEM, kind="stable")
    p = {k: v[order] for k, v in p.items()}
    n, nd = p["iam"].size, int((p["iam"] == cases.DEM).sum())
    whole = capi.Simulation(lib, cfg, p, precision=cases.PREC_FP64)
    mixed = capi.Simulation(lib, cfg, {k: v[:nd] for k, v in p.items()}, precision=cases.PREC_MIXED, capacity=n)
    assert np.array_equal(mixed.insert({k: v[nd:] for k, v in p.items()}), np.arange(nd, n))
    got = []
    for sim in (mixed, whole):
        sim.rebuild()
        sim.rebuild()   # the ghost widths of both handles follow the same h
        sim.step(1)
        a = sim.get()
        got.append({k: a[k].copy() for k in FIELDS})
        sim.close()
    for k in FIELDS:
        assert np.linalg.norm(got[1][k]) > 0 and norm_gap(got[0][k], got[1][k]) <= 1e-9, k


@pytest.mark.parametrize("precision", [cases.PREC_FP64, cases.PREC_MIXED])
def test_contacts_at_the_edge_of_the_search(lib, precision):
    """Pairs of spheres that overlap at distances around 2 max(h), where the
    neighbour predicate decides whether they meet: from 2e-5 of the distance off
    to the last places, both sides of the range in which FP32 decides.  The same
    pairs touch as in the CPU oracle, with the same force (1e-11)."""
    case = cases.dem_settling3d(lattice=(10, 10, 8), spread=0.0, vel_amp=0.0)
    p, R = case.particles, case.cfg["dem_radius"]
    n, h = case.n // 2, p["h"][0]
    rng = np.random.default_rng(2)
    way = rng.standard_normal((n, 3))
    way /= np.linalg.norm(way, axis=1)[:, None]
    off = np.concatenate([[0.0], *([s * 2.0 ** -k for k in range(16, 54)] for s in (1.0, -1.0))])
    gap = 2.0 * h * (1.0 + off[np.arange(n) % off.size])
    q = np.stack(np.unravel_index(np.arange(n), (10, 10, 4)), 1)
    mid = (q + 1.0) * 8.0 * R + rng.uniform(-0.5, 0.5, (n, 3)) * R
    p["r"][:n], p["r"][n:] = mid - 0.5 * gap[:, None] * way, mid + 0.5 * gap[:, None] * way
    p["h"][n:] = h * rng.choice([0.7, 1.0], n)
    p["radius"][:] = 1.1 * h
    p["v"][:] = 0.0
    ora = OracleSim(case.cfg, p)
    ora.step(1)
    want = ora.get()
    sim = capi.Simulation(lib, case.cfg, p, precision=precision)
    sim.step(1)
    got = sim.get()
    touch = np.abs(want["fp"]).sum(axis=1) > 0
    assert 0.2 < touch.mean() < 0.8
    assert np.array_equal(np.abs(got["fp"]).sum(axis=1) > 0, touch)
    assert norm_gap(got["fp"], want["fp"]) <= 1e-11
