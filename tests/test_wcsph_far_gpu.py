"""2-D WCSPH far from the origin: the FP32 build's pair displacements and distances come from the FP64 positions and
are rounded once, so a bed 3e7 m away has the accuracy of one at the origin.

Bar: equal neighbour counts, and per field the FP32 build's distance from the FP64 build after one step at most twice
that of the same bed at the origin (there 1e-5 for state, 1e-4 for rate fields, the suite's bars).  Positions split
into two floats are good to 6e-8 m there, which is 6e-6 of the spacing.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import dam_break_2d
from fluidized_bed_master_b200.params import SPH
from tests.helpers import by_id, rel_l2

pytestmark = pytest.mark.gpu

STATE = ("ux", "uy", "flt_s")
RATE = ("drho", "ftotalx", "ftotaly")


def _errors(shift):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, _ = dam_break_2d(dx=1.0e-2, seed=3)
    rng = np.random.default_rng(4)
    for f in ("ux", "uy"):
        sph[f] = np.where(sph["p_type"] > 0, rng.uniform(-0.1, 0.1, len(sph["x"])), 0.0)
    for f in ("x", "y"):
        sph[f] = sph[f] + shift
    p.freq_filt = 1
    got = []
    for prec in (0, 1):
        q = p.copy()
        q.precision = prec
        with Engine(q, sph, {}) as e:
            e.step(1)
            ids = e.get(SPH, "pid")
            got.append({f: by_id(ids, e.get(SPH, f)) for f in STATE + RATE})
            got[-1]["n"] = by_id(ids, e.neighbors(cap=1)[0])
    assert np.array_equal(got[0]["n"], got[1]["n"]) and got[0]["n"].max() > 15
    return {f: rel_l2(got[0][f], got[1][f]) for f in STATE + RATE}


def test_far_from_the_origin():
    near = _errors(0.0)
    assert all(near[f] <= 1e-5 for f in STATE) and all(near[f] <= 1e-4 for f in RATE)
    far = _errors(3e7)
    assert all(far[f] <= 2 * near[f] for f in near), (near, far)
