"""The FP64 wall pass of Wendland C2 on both sides of the wall count from which it runs in tiles (16,384).

Bar: FP64 build vs the FP64 oracle 1e-9 per field after 2 steps (the suite's bar), the walls' own pressure and
temperature among them.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import box_bed
from fluidized_bed_master_b200.params import SPH
from oracle import Oracle
from tests.helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_fluid,tiled", [(26_000, False), (26_500, True)])
def test_both_forms(n_fluid, tiled):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = box_bed(n_fluid=n_fluid, n_dem=301, lx=0.05, dem_height=0.012, seed=19)
    wall = sph["p_type"] <= 0
    assert (wall.sum() > 16_384) == tiled and abs(wall.sum() - 16_384) < 400
    p.precision = 1
    orc = Oracle(p, sph, dem, threads=8)
    orc.step(2)
    with Engine(p, sph, dem) as eng:
        eng.step(2)
        for f in ("pres", "temp", "rho", "ux", "uz"):
            a, b = by_id(eng.get(SPH, "pid"), eng.get(SPH, f)), by_id(orc.get(SPH, "pid"), orc.get(SPH, f))
            ok = np.isfinite(b)
            assert np.array_equal(ok, np.isfinite(a))
            assert rel_l2(a[ok], b[ok]) <= 1e-9, f
            m = ok & wall   # ids run in the order of the input
            assert rel_l2(a[m], b[m]) <= 1e-9 or not np.linalg.norm(b[m]), f
