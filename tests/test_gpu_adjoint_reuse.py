"""Repeated gradient passes on one handle (-m gpu).  The buffers and replay
graphs of a pass serve the next one of the same form; passes of another length
or tape memory, from a state of more pairs, and after an insertion are opened
anew.  Each must give the gradients of the same pass on a fresh handle: bit for
bit in the position gradients, whose sums have a fixed order; the scalar
gradient is summed by atomics over the warps (1e-9)."""
import numpy as np
import pytest

from sphdem import capi, cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__
    __graft_entry__.build()
    return capi.Library()


def one_pass(sim, r, steps, every, mem, seed):
    sim.set(capi.ParticleBuffers(sim.n, {"r": r}, fields=("r",)), capi.FIELD_R)
    sim.rebuild()
    sim.rebuild()
    sim.adjoint_set_tape_memory(mem)
    sim.adjoint_forward(steps, every)
    g, dr, dv, dvh = sim.adjoint_backward(dL_dr=seed, dL_dv=0.1 * seed)
    return dr, dv, dvh, g.viscosity


@pytest.mark.parametrize("prec", [cases.PREC_FP64, cases.PREC_MIXED])
def test_repeated_passes_equal_fresh_handles(lib, prec):
    case = cases.dambreak2d(dx=0.05)
    rng = np.random.default_rng(9)
    n, fluid = case.n, case.particles["iam"] == cases.SPH
    seed = rng.standard_normal((n, 3)) * fluid[:, None]
    seed[:, 2] = 0.0
    r0 = case.particles["r"].copy()
    squeezed = r0.copy()
    squeezed[fluid, 1] *= 0.6          # more pairs than the first pass's tables hold
    shifted = r0 + 1e-3 * rng.standard_normal(r0.shape) * fluid[:, None] * np.array([1.0, 1.0, 0.0])
    plan = [(r0, 4, 2, -1), (shifted, 4, 2, -1), (r0, 4, 2, -1), (squeezed, 4, 2, -1), (r0, 4, 2, 0), (r0, 3, 2, 0),
            (shifted, 3, 2, 0)]
    kept = capi.Simulation(lib, case.cfg, case.particles, precision=prec)
    start = kept.get()
    state = {k: np.array(start[k]) for k in ("v", "vhat", "f", "dens", "dddt")}
    for r, steps, every, mem in plan:
        got = []
        for sim in (kept, capi.Simulation(lib, case.cfg, case.particles, precision=prec)):
            buf = capi.ParticleBuffers(n, state, fields=tuple(state))
            sim.set(buf, capi.FIELD_V | capi.FIELD_VHAT | capi.FIELD_F | capi.FIELD_DENS | capi.FIELD_DDDT)
            got.append(one_pass(sim, r, steps, every, mem, seed))
            if sim is not kept:
                sim.close()
        for a, b in zip(got[0][:3], got[1][:3]):
            assert np.array_equal(a, b)
        assert abs(got[0][3] - got[1][3]) <= 1e-9 * abs(got[1][3])
    kept.close()


def test_fp64_pair_tables_beyond_the_list_depth(lib):
    """The FP64 gradient takes its pair tables from the neighbour lists, and by a
    bucket scan for a particle whose list is too short: a handle squeezed
    beyond the depth its lists were given at creation gives the gradients of one
    created at the squeezed positions.  Only the order of FP64 sums differs
    (2^-53 a sum of ~100 terms, three steps): 1e-11 of each 2-norm."""
    case = cases.dambreak2d(dx=0.05)
    rng = np.random.default_rng(5)
    n, fluid = case.n, case.particles["iam"] == cases.SPH
    two = np.array([1.0, 1.0, 0.0])
    r = case.particles["r"] + 0.003 * rng.standard_normal((n, 3)) * fluid[:, None] * two
    r[fluid, 1] = 0.02 + 0.3 * (r[fluid, 1] - r[fluid, 1].min())
    v = 0.1 * rng.standard_normal((n, 3)) * fluid[:, None] * two
    seed = rng.standard_normal((n, 3)) * fluid[:, None] * two
    got = []
    for start in (case.particles["r"], r):
        sim = capi.Simulation(lib, case.cfg, dict(case.particles, r=start), precision=cases.PREC_FP64)
        sim.set(capi.ParticleBuffers(n, {"v": v, "vhat": v}, fields=("v", "vhat")), capi.FIELD_V | capi.FIELD_VHAT)
        got.append(one_pass(sim, r, 3, 3, 0, seed))
        sim.close()
    for a, b in zip(*got):
        assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("kind", ["dambreak", "coupled"])
def test_refused_pass_leaves_the_lists(lib, kind):
    """A gradient pass sizes its tables by a count of the present pairs before it
    allocates them.  When the allocation is refused (tapes of 1e8 steps are some
    terabytes) the handle's neighbour lists are the ones of before, and it steps
    on as if nothing had been asked."""
    if kind == "dambreak":
        case = cases.dambreak2d(dx=0.05)
    else:
        case = cases.sediment3d(nx=12, L=0.03, height=0.06, n_dem=60, floor="sphb3", var_h=False)
    sims = [capi.Simulation(lib, case.cfg, case.particles, precision=cases.PREC_MIXED) for _ in range(2)]
    for sim in sims:
        sim.step(2)
    want = sims[0].pairs(capi.PAIRS_SPH)
    with pytest.raises(capi.SphDemError, match="CUDA"):
        sims[0].adjoint_forward(10 ** 8, 10 ** 8)
    got = sims[0].pairs(capi.PAIRS_SPH)
    assert want[1].size > 0 and all(np.array_equal(a, b) for a, b in zip(got, want))
    for sim in sims:
        sim.step(1)
    a, b = (sim.get() for sim in sims)
    # coupled: the Shepard sums' atomics turn FP32 roundings, 2e-7 a step
    tol = 0.0 if kind == "dambreak" else 6e-7
    for k in ("r", "v", "f", "dens"):
        assert np.linalg.norm(a[k] - b[k]) <= tol * np.linalg.norm(b[k]), k


def changed_population(sim, case, kind):
    """Fluid: three particles inserted over the column.  Coupled: a fluid particle
    deleted and a sphere inserted in its slot, so that the count stays and the
    number of spheres does not."""
    p, dx = case.particles, case.cfg["psep"]
    fluid = np.nonzero(p["iam"] == cases.SPH)[0]
    if kind == "fluid":
        block = {k: v[fluid[:3]].copy() for k, v in p.items()}
        block["r"][:, :2] = [[(0.3 + 0.1 * k), p["r"][fluid, 1].max() + 1.1 * dx] for k in range(3)]
        sim.insert(block)
    else:
        gone = int(fluid[np.argmax(p["r"][fluid, 2])])
        sphere = int(np.nonzero(p["iam"] == cases.DEM)[0][0])
        sim.mark_for_deletion([gone])
        sim.rebuild()
        block = {k: v[sphere:sphere + 1].copy() for k, v in p.items()}
        block["r"][0] = p["r"][gone]
        assert list(sim.insert(block)) == [gone]
    sim.rebuild()


@pytest.mark.parametrize("kind,prec", [("fluid", cases.PREC_FP64), ("fluid", cases.PREC_MIXED),
                                       ("coupled", cases.PREC_FP64), ("coupled", cases.PREC_MIXED)])
def test_passes_after_a_changed_population_equal_fresh_handles(lib, kind, prec):
    """Passes of the same form on a handle whose population changed after its first
    pass, then from positions with more pairs than the tables were opened for, and
    back: each as on a handle that has made no pass before.  Fluid
    bit for bit; coupled up to the atomic Shepard sums and the FP32 roundings they
    turn (1e-6 of the largest, as for the two forms of the tables)."""
    if kind == "fluid":
        case = cases.dambreak2d(dx=0.05)
    else:
        case = cases.sediment3d(nx=12, L=0.03, height=0.06, n_dem=60, floor="sphb3", var_h=False)
    steps, every, mem = 4, 2, -1
    rng = np.random.default_rng(3)
    kept = capi.Simulation(lib, case.cfg, case.particles, precision=prec, capacity=case.n + 3)
    kept.adjoint_set_tape_memory(mem)
    kept.adjoint_forward(steps, every)
    kept.adjoint_backward(dL_dr=rng.standard_normal((case.n, 3)))
    changed_population(kept, case, kind)
    model = capi.Simulation(lib, case.cfg, case.particles, precision=prec, capacity=case.n + 3)
    changed_population(model, case, kind)
    start = model.get()
    n, iam = model.n, start["iam"].copy()
    # everything a step starts from (the first drag pass reads the spheres' last fdrag)
    state = {k: np.array(start[k]) for k in ("v", "vhat", "f", "fp", "fv", "fb", "dens", "dddt", "porosity", "dporositydt",
                                             "shep_sum", "fdrag", "fvel", "grad_porosity")}
    r0 = np.array(start["r"])
    model.close()
    # away from zero slip, where the drag law's Jacobian is singular
    moving = (0.02 * (iam == cases.SPH) + 0.05 * (iam == cases.DEM))[:, None]
    state["v"] = moving * rng.standard_normal((n, 3)) * (np.arange(3) < case.cfg["ndim"])
    state["vhat"] = state["v"].copy()
    crowded = r0.copy()
    up, low = (2, 3.0 * case.cfg["psep"]) if kind == "coupled" else (1, 0.0)
    free = iam != cases.SPH_BOUNDARY
    crowded[free, up] = low + 0.6 * (crowded[free, up] - low)
    seed = rng.standard_normal((n, 3)) * (iam != cases.SPH_BOUNDARY)[:, None]
    seed[:, case.cfg["ndim"]:] = 0.0
    for r in (r0, crowded, r0):
        got = []
        fresh = capi.Simulation(lib, case.cfg, case.particles, precision=prec, capacity=case.n + 3)
        changed_population(fresh, case, kind)
        for sim in (kept, fresh):
            assert sim.n == n and np.array_equal(sim.get()["iam"], iam)
            sim.set(capi.ParticleBuffers(n, state, fields=tuple(state)), capi.FIELD_V | capi.FIELD_VHAT | capi.FIELD_F |
                    capi.FIELD_DENS | capi.FIELD_DDDT | capi.FIELD_COUPLING)
            got.append(one_pass(sim, r, steps, every, mem, seed))
        fresh.close()
        for a, b in zip(got[0][:3], got[1][:3]):
            if kind == "fluid":
                assert np.array_equal(a, b)
            else:
                assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
        assert abs(got[0][3] - got[1][3]) <= (1e-9 if kind == "fluid" else 1e-6) * abs(got[1][3])
    kept.close()
