"""The stored operator of the Krylov solve on rows of very different length: a bed thinned out upwards, so that a
warp's rows have from 2 to about 60 entries (whole groups of eight, groups that only some rows fill, odd ends).

Bars as in test_ppe_gpu.py: FP64 build the oracle's iteration counts and 1e-7 per field after 3 steps; FP32 build the
tolerance reached and the pressure within 1e-3.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import box_bed
from fluidized_bed_master_b200.params import PPE_KRYLOV, PPE_PCG, PRECOND_TWO_LEVEL, SPH
from oracle import Oracle
from tests.helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu


def _bed(mode, keep):
    p, sph, _ = box_bed(n_fluid=6_001, n_dem=1, lx=0.02, seed=9)
    p.ppe_mode, p.ppe_tol, p.ppe_max_iter, p.con_solve = mode, 1e-6, 1000, 0
    if mode == PPE_PCG:
        p.kgc_solve = 0
    rng = np.random.default_rng(2)
    z, fluid = sph["z"], sph["p_type"] == 1
    share = 1.0 - (1.0 - keep) * np.clip(z / z[fluid].max(), 0.0, 1.0)
    on = ~fluid | (z < 0.0) | (rng.uniform(size=len(z)) < share)
    return p, {f: v[on] for f, v in sph.items()}


@pytest.mark.parametrize("mode,two_level,keep", [(PPE_PCG, 0, 0.15), (PPE_KRYLOV, 0, 0.15), (PPE_PCG, 1, 0.15),
                                                 (PPE_PCG, 0, 1.0)])
def test_rows_of_mixed_length(mode, two_level, keep):
    from fluidized_bed_master_b200.engine import Engine

    p, sph = _bed(mode, keep)
    orc = None if two_level else Oracle(p, sph, {}, threads=8)
    if two_level:
        p.ppe_precond = PRECOND_TWO_LEVEL
    p64 = p.copy()
    p64.precision = 1
    with Engine(p64, sph, {}) as e64, Engine(p, sph, {}) as e32:
        for _ in range(3):
            for e in (e64, e32):
                e.step(1)
                st = e.stats()
                assert st["ppe_status"] == 0 and st["ppe_rel_residual"] <= 1e-6
            if orc:
                orc.step(1)
                assert e64.stats()["ppe_iters"] == orc.ppe()[0]
        f = lambda e, k: by_id(e.get(SPH, "pid"), e.get(SPH, k))   # noqa: E731
        if orc:
            for k in ("ux", "uz", "pres", "rho"):
                assert rel_l2(f(e64, k), f(orc, k)) <= 1e-7, k
        assert rel_l2(f(e32, "pres"), f(e64, "pres")) <= 1e-3
