"""Sizes at which a pass changes its form: the general neighbour passes on both sides of the particle count up to
which eight lanes work on a particle (18,944), and a wide kernel, with which a sphere has more SPH neighbours than its
list holds (256: the coupling walks the stencil), a buffer particle's lanes fill their queues of eight, and a cell
holds more wall particles than a warp has lanes.

Bar: FP64 build vs the FP64 oracle 1e-9 per field; FP32 vs FP64 build 1e-5 for state, 1e-4 for rate fields after 2
steps (the suite's bars); u against the norm of the vector (ux, uy are the noise of a jittered lattice around zero).
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import box_bed
from fluidized_bed_master_b200.params import DEM, SPH
from oracle import Oracle
from tests.helpers import by_id

pytestmark = pytest.mark.gpu

SMALL_SET = 148 * 4 * 32
SPH_STATE = [("ux", "uy", "uz"), ("m",), ("rho",), ("pres",), ("temp",), ("DEMpor",)]
SPH_RATE = [("ftotalx", "ftotaly", "ftotalz"), ("fpx", "fpy", "fpz")]
DEM_STATE = [("ux", "uy", "uz"), ("DEMpor",), ("flt_s",), ("flt_sd",)]
DEM_RATE = [("Fdx_df", "Fdy_df", "Fdz_df")]


def _worst(a, b, which, groups):
    out = 0.0
    for g in groups:
        x, y = (np.concatenate([by_id(e.get(which, "pid" if which == SPH else "dem_idx"), e.get(which, f)) for f in g])
                for e in (a, b))
        ok = np.isfinite(y)
        assert np.array_equal(ok, np.isfinite(x)), g
        den = np.linalg.norm(y[ok])
        out = max(out, np.linalg.norm(x[ok] - y[ok]) / den if den else np.linalg.norm(x[ok]))
    return out


def _compare(p, sph, dem):
    from fluidized_bed_master_b200.engine import Engine

    orc = Oracle(p, sph, dem, threads=8)
    orc.step(2)
    p64 = p.copy()
    p64.precision = 1
    with Engine(p64, sph, dem) as e64, Engine(p, sph, dem) as e32:
        e64.step(2)
        e32.step(2)
        assert _worst(e64, orc, SPH, SPH_STATE + SPH_RATE) <= 1e-9
        assert _worst(e64, orc, DEM, DEM_STATE + DEM_RATE) <= 1e-9
        assert _worst(e32, e64, SPH, SPH_STATE) <= 1e-5
        assert _worst(e32, e64, SPH, SPH_RATE) <= 1e-4
        assert _worst(e32, e64, DEM, DEM_STATE) <= 1e-5
        assert _worst(e32, e64, DEM, DEM_RATE) <= 1e-4


@pytest.mark.parametrize("kernel,n_fluid,small", [(4, 9_001, True), (5, 9_001, True), (4, 9_301, False),
                                                  (5, 9_301, False)])
def test_lanes_per_particle(kernel, n_fluid, small):
    p, sph, dem = box_bed(n_fluid=n_fluid, n_dem=401, dem_height=0.012, lx=0.02, seed=13)
    p.kernel_type = kernel
    assert (len(sph["x"]) <= SMALL_SET) == small
    _compare(p, sph, dem)


@pytest.mark.parametrize("kernel,n_fluid", [(3, 4_001), (5, 4_001), (3, 9_301), (5, 9_301)])
def test_wide_kernel(kernel, n_fluid):
    p, sph, dem = box_bed(n_fluid=n_fluid, n_dem=101, dem_height=0.012, lx=0.02, seed=17)
    p.kernel_type = kernel
    p.h_over_dx *= 1.7
    sph["h"] = sph["h"] * 1.7
    dem["h"] = dem["h"] * 1.7
    d2 = sum((sph[c][None] - dem[c][:, None]) ** 2 for c in "xyz")
    assert ((d2 < (p.kappa * dem["h"][:, None]) ** 2).sum(1) > 256).any()
    _compare(p, sph, dem)
