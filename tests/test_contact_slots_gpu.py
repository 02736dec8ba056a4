"""Contact history slots when a sphere loses one partner and meets another in the same step: the new contact takes the
first slot free at the start of the step, never the one given up in it.

Bar: partner ids exact slot by slot against the oracle; their springs and the spheres' state to 1e-9 (the suite's bar
for FP64).
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import _dem_arrays, box_bed
from fluidized_bed_master_b200.params import DEM
from oracle import Oracle
from tests.helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu


def _bed(seed, v):
    """2,744 spheres that just touch, each with a random velocity."""
    p, sph, _ = box_bed(n_fluid=4_001, n_dem=1, lx=0.02, seed=5)
    p.con_solve = 0
    p.precision = 1
    rng = np.random.default_rng(seed)
    r = 0.5e-3
    pos = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3) * (2.0 * r) + 2.5e-3
    pos = pos + rng.uniform(-0.02 * r, 0.02 * r, pos.shape)
    dem = _dem_arrays(pos, np.full(len(pos), r), 2500.0, float(sph["h"][0]), 350.0)
    for f in ("ux", "uy", "uz"):
        dem[f] = rng.uniform(-v, v, len(pos))
    return p, sph, dem


@pytest.mark.parametrize("seed,v", [(1, 0.5), (2, 2.0)])
def test_release_and_new_contact_in_one_step(seed, v):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(seed, v)
    orc = Oracle(p, sph, dem, threads=8)
    both, prev = 0, None
    with Engine(p, sph, dem) as eng:
        for _ in range(5):
            eng.step(1)
            orc.step(1)
            ie, io = eng.get(DEM, "dem_idx"), orc.get(DEM, "dem_idx")
            he, ho = eng.history(), orc.history()
            a, b = by_id(ie, he[0]), by_id(io, ho[0]).astype(int)
            held = b >= 1
            assert np.array_equal(np.where(a >= 1, a, 0), np.where(held, b, 0))
            assert rel_l2(by_id(ie, he[1])[held], by_id(io, ho[1])[held]) <= 1e-9
            for f in ("x", "ux", "uy", "uz", "wx", "ftotalx", "ftotalz"):
                assert rel_l2(by_id(ie, eng.get(DEM, f)), by_id(io, orc.get(DEM, f))) <= 1e-9, f
            if prev is not None:
                both += sum(bool(set(p0[p0 >= 1]) - set(p1[p1 >= 1]) and set(p1[p1 >= 1]) - set(p0[p0 >= 1]))
                            for p0, p1 in zip(prev, b))
            prev = b
    assert both > 100
