"""The fused 2-D WCSPH step (Wendland C2, no gradient correction, no delta-SPH) against the FP64 oracle at the places
where it can go wrong: every lane count, XSPH behind it, each force switched off, filter steps, a tank far from the
origin (the records' split positions), and the list's rows at the edge of the grid.

Bar: FP64 1e-9 per field and lists bit-exact; FP32 1e-5 per field, pressure and rates against their largest value
(the bars of the dam break tests).
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import dam_break_2d
from fluidized_bed_master_b200.params import SPH
from oracle import Oracle
from tests.helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu

STATE = ["x", "y", "ux", "uy", "rho"]
MAXED = ["pres", "drho", "ftotalx", "ftotaly"]


def _bed(xsph=0, off=0.0, **sw):
    p, sph, _ = dam_break_2d(dx=2.0e-2, seed=3, tank=(0.82, 0.5), column=(0.2, 0.3))
    p.xsph_solve, p.freq_filt = xsph, 3
    for k, v in sw.items():
        setattr(p, k, v)
    sph["x"] = sph["x"] + off
    sph["y"] = sph["y"] - 2 * off
    return p, sph


@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("kw", [dict(), dict(xsph=1), dict(off=40.0), dict(fva_solve=0), dict(fp_solve=0),
                                dict(fv_solve=0, fg_solve=0)])
def test_fused_step_vs_oracle(kw, lanes):
    from fluidized_bed_master_b200.engine import Engine

    p, sph = _bed(**kw)
    p.w_lanes = lanes
    orc = Oracle(p, sph, {}, threads=4)
    orc.step(7)
    ido = orc.get(SPH, "pid")
    for prec in (1, 0):
        q = p.copy()
        q.precision = prec
        with Engine(q, sph, {}) as eng:
            eng.step(7)
            ide = eng.get(SPH, "pid")
            assert np.array_equal(ide, ido)
            ce, le = eng.neighbors(cap=64)
            co, lo = orc.neighbors(cap=64)
            assert np.array_equal(ce, co) and np.array_equal(le, lo)
            for f in STATE + ["flt_s"]:
                assert rel_l2(by_id(ide, eng.get(SPH, f)), by_id(ido, orc.get(SPH, f))) <= (1e-9 if prec else 1e-5), f
            for f in MAXED:
                a, b = by_id(ide, eng.get(SPH, f)), by_id(ido, orc.get(SPH, f))
                assert np.abs(a - b).max() <= (1e-9 if prec else 1e-5) * max(np.abs(b).max(), 1e-300), f
