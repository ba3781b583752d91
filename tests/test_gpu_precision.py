"""Mixed precision against the FP64 path over 1000 steps (-m gpu).

Bar: max |rho_mixed - rho_fp64| / rho0 <= 1e-4 and
max |f_mixed - f_fp64| / max |f_fp64| <= 1e-4 (maxima over the fluid
particles), checked every 100 steps from the same input.

- The 2D dam break (20,000 fluid particles + 3-layer walls, dx = 0.01):
  the bar holds at every checkpoint to step 1000.
- The coupled solver (VAR_H_CORRECTION, porosity-weighted Tait EOS, Morris
  viscosity, porosity / Shepard / drag passes) on the 1/16 periodic sub-box
  of the coupled sedimentation workload with a single DEM sphere and a floor
  of three fixed sphBoundary layers: the bar holds at every checkpoint to
  step 1000.
- The coupled workload at its full size (1,080,400 particles): every 100
  steps along a 1000-step mixed run, an FP64 handle started from the mixed
  handle's state takes the same step; the two agree to the bar in rho and f
  at every checkpoint.  This bounds the mixed arithmetic's own error at each
  point of the run, apart from the flow's amplification of earlier
  differences (below).
- The coupled workload as configured (the same sub-box with its 3,125 DEM
  spheres and the repulsive boundary floor): the bar holds at the first
  checkpoint, and the runs then separate at the rate the sedimenting
  suspension amplifies any perturbation.  The FP64 path run from inputs one
  bit apart (the x coordinate of one sphere moved to the next double)
  separates just as far by step 1000, so no arithmetic meets a pointwise
  1000-step bar on this flow.  The test asserts the first-checkpoint bar;
  that the one-bit FP64 runs differ by more than the bar at step 1000; that
  the mixed-vs-FP64 difference grows at the rate of the one-bit difference
  (slopes of log10 of the density difference per step, fitted where each lies
  between its start and 1e-3, within a factor of two of each other); and that
  the mixed difference saturates below 0.5 rho0, the size of the flow's own
  density fluctuations.
"""
import numpy as np
import pytest

from sphdem import capi, cases

pytestmark = pytest.mark.gpu

NSTEPS = 1000
EVERY = 100
TOL = 1e-4
MASK = capi.FIELD_DENS | capi.FIELD_F | capi.FIELD_IAM


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__
    __graft_entry__.build()
    return capi.Library()


def _err(a, b, rho0):
    """max |d rho| / rho0 and max |d f| / max |f| over the fluid particles."""
    iam = b["iam"]
    fl = (iam == cases.SPH) | (iam == cases.SPH_BOUNDARY)
    e_rho = float(np.abs(a["dens"][fl] - b["dens"][fl]).max() / rho0)
    e_f = float(np.abs(a["f"][fl] - b["f"][fl]).max() / np.abs(b["f"][fl]).max())
    return e_rho, e_f


def _against_fp64(lib, case, others):
    """Step an FP64 handle and the `others` (name -> (precision, particles))
    together; per checkpoint, each other's errors against the FP64 handle."""
    ref = capi.Simulation(lib, case.cfg, case.particles, precision=cases.PREC_FP64)
    sims = {k: capi.Simulation(lib, case.cfg, ps, precision=p) for k, (p, ps) in others.items()}
    rows = {k: [] for k in others}
    try:
        for c in range(NSTEPS // EVERY):
            ref.step(EVERY)
            b = ref.get(MASK)
            for k, sim in sims.items():
                sim.step(EVERY)
                rows[k].append((EVERY * (c + 1),) + _err(sim.get(MASK), b, case.cfg["dens"]))
    finally:
        ref.close()
        for sim in sims.values():
            sim.close()
    for k, r in rows.items():
        for s, e_rho, e_f in r:
            print(f"{case.name} {k} step {s}: max|drho|/rho0 {e_rho:.2e}  max|df|/max|f| {e_f:.2e}")
    return rows


def test_dambreak_mixed_vs_fp64_1000_steps(lib):
    case = cases.dambreak2d(dx=0.01, nsteps=NSTEPS)
    rows = _against_fp64(lib, case, {"mixed": (cases.PREC_MIXED, case.particles)})["mixed"]
    for s, e_rho, e_f in rows:
        assert e_rho <= TOL and e_f <= TOL, f"step {s}: {e_rho:.2e} {e_f:.2e}"


# the state a step starts from: the fields creation takes, then the forces,
# continuity rates, lagged DEM drag and energy rates, and the step globals
STATE_INIT = ("iam", "r", "v", "vhat", "mass", "dens", "h", "radius", "norm1", "norm2", "norm3")
STATE_SET = ("f", "fp", "fv", "fb", "dddt", "fdrag", "u", "e_visc", "dudt", "de_visc_dt")


def _clone(lib, cfg, src, precision):
    """A new handle of `precision` holding src's state, as an exact restart does."""
    a = src.get(capi.FIELD_ALL)
    dst = capi.Simulation(lib, cfg, {k: np.array(a[k]) for k in STATE_INIT}, precision=precision)
    buf = dst.get(capi.FIELD_ALL)
    for k in STATE_SET:
        buf[k][...] = a[k]
    dst.set(buf, capi.FIELD_F | capi.FIELD_DDDT | capi.FIELD_COUPLING | capi.FIELD_ENERGY)
    dst.set_globals(src.globals())
    return dst


def test_coupled_full_size_one_step_error_along_1000_steps(lib):
    """The 1.08M coupled workload: at every 100th step of a 1000-step mixed
    run, one step from the mixed state in FP64 against the mixed step."""
    case = cases.workload("sediment3d")
    rho0 = case.cfg["dens"]
    m = capi.Simulation(lib, case.cfg, case.particles, precision=cases.PREC_MIXED)
    worst = (0.0, 0.0)
    try:
        for c in range(NSTEPS // EVERY):
            m.step(EVERY - 1)
            f = _clone(lib, case.cfg, m, cases.PREC_FP64)
            try:
                m.step(1)
                f.step(1)
                e_rho, e_f = _err(m.get(MASK), f.get(MASK), rho0)
            finally:
                f.close()
            print(f"step {EVERY * (c + 1)}: one step mixed vs FP64 from the same state: "
                  f"max|drho|/rho0 {e_rho:.2e}  max|df|/max|f| {e_f:.2e}")
            worst = (max(worst[0], e_rho), max(worst[1], e_f))
            assert e_rho <= TOL and e_f <= TOL, f"step {EVERY * (c + 1)}: {e_rho:.2e} {e_f:.2e}"
    finally:
        m.close()
    print(f"worst over the run: {worst[0]:.2e} {worst[1]:.2e}")


def _coupled_box(floor="boundary", n_dem=3125):
    return cases.sediment3d(nx=20, L=0.05, height=0.4, n_dem=n_dem, seed=3, nsteps=NSTEPS, floor=floor)


def test_coupled_fluid_mixed_vs_fp64_1000_steps(lib):
    case = _coupled_box(floor="sphb3", n_dem=1)
    case.name = "coupled fluid"
    rows = _against_fp64(lib, case, {"mixed": (cases.PREC_MIXED, case.particles)})["mixed"]
    for s, e_rho, e_f in rows:
        assert e_rho <= TOL and e_f <= TOL, f"step {s}: {e_rho:.2e} {e_f:.2e}"


def test_coupled_suspension_against_fp64_one_bit_divergence(lib):
    case = _coupled_box()
    case.name = "suspension"
    parts = {k: np.array(v) for k, v in case.particles.items()}
    i = int(np.nonzero(parts["iam"] == cases.DEM)[0][0])
    parts["r"][i, 0] = np.nextafter(parts["r"][i, 0], 1.0)
    rows = _against_fp64(lib, case, {"mixed": (cases.PREC_MIXED, case.particles),
                                     "fp64 one bit": (cases.PREC_FP64, parts)})
    mixed, onebit = rows["mixed"], rows["fp64 one bit"]
    s, e_rho, e_f = mixed[0]
    assert e_rho <= TOL and e_f <= TOL, f"step {s}: {e_rho:.2e} {e_f:.2e}"
    # the FP64 path does not reproduce itself to the bar over 1000 steps
    assert onebit[-1][1] > TOL

    def slope(rows):
        pts = [(s, np.log10(e)) for s, e, _ in rows if 0.0 < e < 1e-3]
        assert len(pts) >= 2, rows
        x, y = np.array(pts).T
        return float(np.polyfit(x, y, 1)[0])

    k_mixed, k_onebit = slope(mixed), slope(onebit)
    print(f"growth of log10 max|drho|/rho0 per step: mixed {k_mixed:.4f}, fp64 one bit {k_onebit:.4f}")
    assert 0.5 <= k_mixed / k_onebit <= 2.0
    assert max(e for _, e, _ in mixed) < 0.5


def _pairs_far_apart(nd, h, seed):
    """Pairs of fluid particles at r = 0.3 .. 1.98 h, as many in each shell as a
    uniform fluid has, each pair alone, with a mass of FP32's own numbers, random
    densities and no velocity."""
    rng = np.random.default_rng(seed)
    cfg = cases.dambreak2d(dx=0.1).cfg
    side = 16 if nd == 2 else 7
    ext = side * 7.0 * h
    cfg.update(ndim=nd, psep=h / 1.3, h=h, rmax=[ext] * nd + [0.0] * (3 - nd), domain_min=[-4 * h] * nd + [0.0] * (3 - nd),
               domain_max=[ext + 4 * h] * nd + [0.0] * (3 - nd), gravity_sph=[0.0] * 3, maxdt=1e-12)
    q = np.stack(np.unravel_index(np.arange(side ** nd), (side,) * nd), 1)
    m = len(q)
    way = rng.standard_normal((m, nd))
    way /= np.linalg.norm(way, axis=1)[:, None]
    p = cases._empty_particles(2 * m)
    mid = (q + 0.5 + rng.uniform(-0.1, 0.1, q.shape)) * 7.0 * h
    gap = 0.5 * h * rng.uniform(0.3 ** nd, 1.98 ** nd, (m, 1)) ** (1.0 / nd) * way
    p["r"][:m, :nd], p["r"][m:, :nd] = mid + gap, mid - gap
    p["mass"][:] = 2.0 ** np.round(np.log2(1000.0 * (h / 1.3) ** nd))
    p["dens"][:] = 1000.0 * rng.uniform(1.01, 1.05, 2 * m)
    p["h"][:] = h
    return cfg, p


@pytest.mark.parametrize("nd", [2, 3])
def test_kernel_gradient_has_no_error_of_one_sign(lib, nd):
    """The moment sum of the pair forces, sum f.r -- what a pressure gradient comes
    from -- of the mixed path against FP64, for 40 values of a constant h (numbers of
    FP32's own, so that the bucket size 2 h is exact in the displacements).  A kernel
    keeps this moment whatever its h, so the rounding of 1/h drops out where factor
    and argument of F(r, h) share it; left are the rounding of cF (uniform in half
    an ulp: rms 2.5e-8) and the pairs' own roundings by the root of their number
    (2e-8): 3.2e-8 rms, and an rms of 40 values strays by a ninth: bound 5e-8.  With
    cF of the FP64 h next to (2 - r/h)^3 of the FP32 one it is 1.1e-7 in 2D and
    1.3e-7 in 3D."""
    rng = np.random.default_rng(11)
    shift = []
    for k in range(40):
        h = float(np.float32(10.0 ** rng.uniform(-3.0, -1.0)))
        cfg, p = _pairs_far_apart(nd, h, k)
        f = []
        for prec in (cases.PREC_FP64, cases.PREC_MIXED):
            sim = capi.Simulation(lib, cfg, p, precision=prec)
            sim.step(1)
            f.append(sim.get()["f"])
            sim.close()
        m = len(p["h"]) // 2
        d = p["r"][:m] - p["r"][m:]
        moment = [np.einsum("ij,ij->", x[:m] - x[m:], d) for x in f]
        shift.append(moment[1] / moment[0] - 1.0)
    assert np.sqrt(np.mean(np.square(shift))) <= 5e-8
