"""sphdem_step(h, n) against n calls of sphdem_step(h, 1): a call's later steps
keep its SPH order and neighbour list, single calls build them every time; every
field, the order and the lists are bit-identical, with step graphs and without,
on one stream and two, and after the caller moved particles between two calls.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import bed2d_batch, box_bed, isph_column, spouted_bed
from fluidized_bed_master_b200.params import DEM, PRECOND_TWO_LEVEL, SPH, WARM_PROJECT

pytestmark = pytest.mark.gpu

SPH_F = ["pid", "cell", "x", "ux", "uy", "uz", "m", "rho", "pres", "temp", "DEMpor", "dDEMpor", "flt_s", "ftotalx",
         "fpz", "dtemp"]
DEM_F = ["dem_idx", "x", "y", "z", "ux", "uz", "wy", "temp", "ftotalz", "Q_sd"]


def _cfg(kind):
    rows = None
    if kind == "spouted":
        p, sph, dem = spouted_bed(dx=2.0e-3, n_dem=200, r_dem=1.0e-3, seed=3, u_dem=0.05)
    elif kind == "bed2d":
        p, sph, dem, rows, _ = bed2d_batch(n_beds=3, n_min=1500, n_max=3000, seed=5)
    elif kind == "column":
        p, sph, dem = isph_column(dx=1.0e-2, seed=2)
    else:
        p, sph, dem = box_bed(n_fluid=6_001, n_dem=601, dem_height=0.02, lx=0.03, seed=9)
        p.freq_filt = 3
        if kind == "pcg":
            p.ppe_mode, p.kgc_solve, p.ppe_precond, p.warm_start, p.warm_hist = 2, 0, PRECOND_TWO_LEVEL, WARM_PROJECT, 2
        if kind == "noxsph":
            p.xsph_solve = 0
    return p, sph, dem, rows


def _same(a, b):
    for which, names in ((SPH, SPH_F), (DEM, DEM_F)):
        if which == DEM and a.nd == 0:
            continue
        for f in names:
            assert np.array_equal(a.get(which, f), b.get(which, f), equal_nan=True), f
    (ca, la), (cb, lb) = a.neighbors(cap=160), b.neighbors(cap=160)
    assert np.array_equal(ca, cb) and np.array_equal(la, lb)


@pytest.mark.parametrize("kind,precision", [("box", 0), ("box", 1), ("noxsph", 0), ("spouted", 0), ("bed2d", 0),
                                            ("column", 0), ("pcg", 0)])
def test_steps_in_one_call(kind, precision):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem, rows = _cfg(kind)
    p.precision = precision
    with Engine(p, sph, dem, beds=rows) as a, Engine(p, sph, dem, beds=rows) as b:
        for n in (1, 2, 5, 4):
            a.step(n)
            for _ in range(n):
                b.step(1)
        _same(a, b)
        # positions replaced between two calls: the next call's first step sorts and lists again
        for e in (a, b):
            x = e.get(SPH, "x")
            e.set(SPH, "x", x + np.where(e.get(SPH, "z") > 0.01, 3e-3, 0.0))
        a.step(3)
        for _ in range(3):
            b.step(1)
        _same(a, b)


@pytest.mark.parametrize("graphs,concurrent", [(False, True), (True, False), (False, False)])
def test_steps_in_one_call_without_graphs_or_streams(graphs, concurrent):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem, _ = _cfg("box")
    with Engine(p, sph, dem) as a, Engine(p, sph, dem) as b:
        a.set_graphs(graphs)
        a.set_concurrency(concurrent)
        a.step(7)
        for _ in range(7):
            b.step(1)
        _same(a, b)
