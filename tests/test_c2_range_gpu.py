"""Wendland C2 with particles outside the fixed-point range of the FP32 build's positions: its neighbour passes take
such pairs from the double positions, and its wall pass mixes candidates of both kinds in one wall's sums.

Bars as in test_pair_records_gpu.py: FP32 vs FP64 build 1e-5 for state, 1e-4 for rate fields after 3 steps; the walls'
own pressure 1e-5.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.params import DEM, SPH
from tests.helpers import by_id, rel_l2
from tests.test_pair_records_gpu import RATE, STATE, _bed, _worst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heat", [0, 1])
def test_moved_fragment(heat):
    """The upper part of the bed moved sideways by three box widths: clamped into the last column of cells beside
    walls whose other candidates are in range."""
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(3, heat, 0, 0)
    p64 = p.copy()
    p64.precision = 1
    with Engine(p64, sph, dem) as e64, Engine(p, sph, dem) as e32:
        for e in (e64, e32):
            x, z = e.get(SPH, "x"), e.get(SPH, "z")
            e.set(SPH, "x", x + np.where((z > 0.012) & (x > 0.012), 0.15, 0.0))
            e.step(3)
        assert np.array_equal(np.sort(e64.neighbors(cap=1)[0]), np.sort(e32.neighbors(cap=1)[0]))
        assert e64.get(SPH, "x").max() > 0.15
        assert _worst(e32, e64, STATE) <= 1e-5
        assert _worst(e32, e64, RATE) <= 1e-4
        ids, pres = ([by_id(e.get(SPH, "pid"), e.get(SPH, f)) for e in (e32, e64)] for f in ("p_type", "pres"))
        assert rel_l2(pres[0][ids[0] <= 0], pres[1][ids[1] <= 0]) <= 1e-5
        assert np.array_equal(e64.get(DEM, "dem_idx"), e32.get(DEM, "dem_idx"))
