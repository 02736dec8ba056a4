"""Wendland C2 passes with particles of negative mass or density (a negative m / rho, which the volume records cannot
hold), kept from step to step by rho_type 0: every sum takes them with their sign.

Bar: FP64 build vs the FP64 oracle 1e-9 per field; for negative masses also FP32 vs FP64 build, 1e-5 for state, 1e-4
for rate fields after 2 steps (the suite's bars).  With negative densities the diagonal of a pressure row nearly
cancels (2e10 Pa against a median of 360), which FP32 sums of any order cannot hold.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.params import SPH
from oracle import Oracle
from tests.test_pair_records_gpu import RATE, STATE, _bed, _worst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["m", "rho"])
def test_negative_volumes(field):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(3, 1, 0, 0)
    p.rho_type = 0
    p.xsph_solve = 1
    rng = np.random.default_rng(5)
    fluid = np.flatnonzero((sph["p_type"] == 1) & (sph["z"] > 0.002) & (sph["z"] < p.obc_L3 - 0.002))
    pick = rng.choice(fluid, 25, replace=False)
    sph[field] = sph[field].copy()
    sph[field][pick] *= -0.3
    sph["ux"] = sph["ux"] + rng.uniform(-0.05, 0.05, len(sph["ux"])) * (sph["p_type"] == 1)
    orc = Oracle(p, sph, dem, threads=8)
    orc.step(2)
    p64 = p.copy()
    p64.precision = 1
    with Engine(p64, sph, dem) as e64, Engine(p, sph, dem) as e32:
        e64.step(2)
        e32.step(2)
        assert np.isfinite(orc.get(SPH, "ux")).all()
        assert _worst(e64, orc, STATE + RATE) <= 1e-9
        if field == "m":
            assert _worst(e32, e64, STATE) <= 1e-5
            assert _worst(e32, e64, RATE) <= 1e-4
