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
