"""A whole step against the same step phase by phase (-m gpu).  A whole step
takes the elementwise work of neighbouring phases and hooks in the passes that
precede its two rebuilds; the phase-level calls run each by itself.  Both
evaluate the same device functions, so the states are equal bit for bit; where
fluid and spheres are coupled, up to the order of the atomic Shepard sums and
the FP32 roundings it turns (2e-7 of a field's 2-norm in mixed precision, 1e-12
in FP64).  Covered: one block and several, bucket grids on both sides of the
single-block prefix sum (131,072 buckets), hooks (gravity, planar walls, freeze),
density re-initialisation, particles that leave the domain, DEM without fluid."""
import copy

import numpy as np
import pytest

from sphdem import capi, cases

pytestmark = pytest.mark.gpu

FIELDS = ("r", "v", "vhat", "f", "fp", "fv", "fb", "dens", "h", "dddt", "omega", "fdrag")


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__
    __graft_entry__.build()
    return capi.Library()


def run(lib, cfg, p, prec, steps, whole):
    sim = capi.Simulation(lib, cfg, p, precision=prec)
    for _ in range(steps):
        if whole:
            sim.step(1)
        else:
            for ph in range(7):
                sim.phase(ph)
    a, g = sim.get(), sim.globals()
    out = {k: np.array(a[k]) for k in FIELDS}
    scalars = {k: getattr(g, k) for k, _ in g._fields_ if isinstance(getattr(g, k), (int, float))}
    sim.close()
    return out, scalars


@pytest.mark.parametrize("prec", [cases.PREC_FP64, cases.PREC_MIXED])
@pytest.mark.parametrize("kind", ["dambreak2d_small", "dambreak2d_own_small", "wide", "lost", "dem_small", "sediment3d_small",
                                  "sediment3d_reinit_small", "sediment3d_block_small"])
def test_whole_step_equals_phases(lib, kind, prec):
    w = cases.workload(kind if "small" in kind else "dambreak2d_small")
    cfg, p = copy.deepcopy(w.cfg), {k: np.array(v) for k, v in w.particles.items()}
    dx = cfg["psep"]
    if kind == "wide":
        cfg["domain_min"], cfg["domain_max"] = [-1200 * dx] * 2 + [0.0], [1200 * dx] * 2 + [0.0]
    if kind == "lost":
        top = p["r"][p["iam"] == cases.SPH, 1].max()
        cfg["domain_max"] = [cfg["domain_max"][0], top - 0.5 * dx, 0.0]
    coupled = kind.startswith("sediment")
    steps = 1 if coupled else 3
    (a, ga), (b, gb) = (run(lib, cfg, p, prec, steps, whole) for whole in (True, False))
    if not coupled:
        assert ga == gb
    assert kind != "lost" or ga["n_deleted"] > 0
    tol = 0.0 if not coupled else (1e-12 if prec == cases.PREC_FP64 else 2e-7)
    for k in FIELDS:
        assert np.linalg.norm(a[k] - b[k]) <= tol * np.linalg.norm(b[k]), k
