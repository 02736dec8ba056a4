"""The neighbour sums over position + volume records, in every form they take:
the two kernels fixed at compile time (Wendland C2 and C6) and one that is not,
heat on and off, artificial viscosity (the form that reads m_j and rho_j), and
the particles that a pass cannot take from the record alone: p_type 1000, and
positions outside the fixed-point range of the FP32 build.

Bar: FP64 build vs the FP64 oracle 1e-9 per field (the suite's bar for sums
regrouped in double); FP32 vs FP64 build 1e-5 for state, 1e-4 for rate fields
after 3 steps (the suite's FP32 bars).  ux, uy and the rates along them are
the noise of a jittered lattice around zero: their bar is against the norm of
the vector.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import box_bed
from fluidized_bed_master_b200.params import DEM, SPH
from oracle import Oracle
from tests.helpers import by_id

pytestmark = pytest.mark.gpu

STATE = [("ux", "uy", "uz"), ("m",), ("rho",), ("pres",), ("temp",), ("DEMpor",), ("flt_s",)]
RATE = [("ftotalx", "ftotaly", "ftotalz"), ("fpx", "fpy", "fpz"), ("pgfx", "pgfy", "pgfz"), ("dtemp",)]


def _fields(eng, names):
    ids = eng.get(SPH, "pid")
    return np.concatenate([by_id(ids, eng.get(SPH, f)) for f in names])


def _worst(a, b, groups):
    out = 0.0
    for g in groups:
        x, y = _fields(a, g), _fields(b, g)
        assert np.array_equal(np.isfinite(x), np.isfinite(y)), g
        ok = np.isfinite(y)
        den = np.linalg.norm(y[ok])
        out = max(out, np.linalg.norm(x[ok] - y[ok]) / den if den else np.linalg.norm(x[ok]))
    return out


def _bed(kernel, heat, fva, special):
    p, sph, dem = box_bed(n_fluid=4_001, n_dem=401, dem_height=0.012, lx=0.02, seed=11)
    p.kernel_type, p.con_solve, p.fva_solve = kernel, heat, fva
    if special:
        rng = np.random.default_rng(3)
        sph["p_type"] = sph["p_type"].copy()
        fluid = np.flatnonzero((sph["p_type"] == 1) & (sph["z"] > 0.002) & (sph["z"] < p.obc_L3 - 0.002))
        sph["p_type"][rng.choice(fluid, 40, replace=False)] = 1000
    return p, sph, dem


@pytest.mark.parametrize("kernel,heat,fva,special", [(3, 1, 0, 0), (3, 0, 0, 1), (5, 1, 0, 1), (5, 0, 0, 0),
                                                     (4, 1, 0, 1), (3, 1, 1, 1), (5, 0, 1, 0)])
def test_forms_vs_oracle(kernel, heat, fva, special):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(kernel, heat, fva, special)
    orc = Oracle(p, sph, dem, threads=8)
    orc.step(3)
    p64 = p.copy()
    p64.precision = 1
    with Engine(p64, sph, dem) as e64, Engine(p, sph, dem) as e32:
        e64.step(3)
        e32.step(3)
        assert _worst(e64, orc, STATE + RATE) <= 1e-9
        assert _worst(e32, e64, STATE) <= 1e-5
        assert _worst(e32, e64, RATE) <= 1e-4


@pytest.mark.parametrize("kernel", [5, 4])
def test_particles_outside_the_fixed_point_range(kernel):
    """The upper part of the bed moved sideways by three box widths: clamped into the last column of cells, outside
    the range of the FP32 build's fixed-point positions, with neighbours among themselves."""
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(kernel, 1, 0, 0)
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
        assert np.array_equal(e64.get(DEM, "dem_idx"), e32.get(DEM, "dem_idx"))
