"""The contact pass over the list of spheres in range: polydisperse packings in which a large sphere has more spheres
in its search range than the list holds (it walks its stencil), spheres in contact from the start, and a sphere alone.

Bar: contact partners and springs' partners exact against the oracle, FP64 fields to 1e-9 (the suite's bar).
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import _dem_arrays, box_bed
from fluidized_bed_master_b200.params import DEM
from oracle import Oracle
from tests.helpers import by_id, history_map, rel_l2

pytestmark = pytest.mark.gpu

FIELDS = ["x", "y", "z", "ux", "uy", "uz", "wx", "wy", "wz", "temp", "temp1", "ftotalx", "ftotaly", "ftotalz"]


def _bed(big, n_small, heat):
    p, sph, _ = box_bed(n_fluid=4_001, n_dem=1, lx=0.02, seed=5)
    p.con_solve = heat
    rng = np.random.default_rng(7)
    s = 1.02e-3
    g = np.stack(np.meshgrid(*[np.arange(13)] * 3, indexing="ij"), -1).reshape(-1, 3) * s + 2.0e-3
    c = np.array([8.0e-3, 8.0e-3, 8.0e-3])
    d = np.linalg.norm(g - c, axis=1)
    g = g[d > big + 0.5e-3]
    g = g[np.argsort(np.linalg.norm(g - c, axis=1), kind="stable")][:n_small]
    pos = np.concatenate([c[None], g])
    rad = np.r_[big, np.full(len(g), 0.515e-3) * rng.uniform(0.97, 1.0, len(g))]
    dem = _dem_arrays(pos, rad, 2500.0, float(sph["h"][0]), 350.0)
    for f in ("ux", "uy", "uz", "wx", "wy", "wz"):
        dem[f] = rng.uniform(-0.05, 0.05, len(rad))
    return p, sph, dem


@pytest.mark.parametrize("big,n_small,heat", [(0.9e-3, 200, 1), (1.0e-3, 400, 0), (0.515e-3, 60, 1), (0.6e-3, 0, 1)])
def test_contact_over_the_list(big, n_small, heat):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(big, n_small, heat)
    p.precision = 1
    orc = Oracle(p, sph, dem, threads=4)
    with Engine(p, sph, dem) as eng:
        for n in (1, 4):
            eng.step(n)
            orc.step(n)
            ie, io = eng.get(DEM, "dem_idx"), orc.get(DEM, "dem_idx")
            assert np.array_equal(ie, io)
            for f in FIELDS:
                a, b = by_id(ie, eng.get(DEM, f)), by_id(io, orc.get(DEM, f))
                ok = np.isfinite(b)
                assert np.array_equal(ok, np.isfinite(a)), f
                assert rel_l2(a[ok], b[ok]) <= 1e-9, f
            he, ho = history_map(*eng.history()), history_map(*orc.history())
            assert [sorted(m) for m in he] == [sorted(m) for m in ho]
