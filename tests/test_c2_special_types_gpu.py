"""Wendland C2 with heat and p_type 1000 particles, without artificial viscosity: the passes over position + volume
records (not the general ones) take the marked pairs from the tagged records.

Bars as in test_pair_records_gpu.py: FP64 build vs the FP64 oracle 1e-9 per field, FP32 vs FP64 build 1e-5 for state
and 1e-4 for rate fields, after 3 steps and over a step of the Shepard filter.
"""
import pytest

from oracle import Oracle
from tests.test_pair_records_gpu import RATE, STATE, _bed, _worst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heat,kgc,freq_filt", [(1, 1, 40), (1, 0, 2), (0, 1, 1)])
def test_marked_pairs(heat, kgc, freq_filt):
    from fluidized_bed_master_b200.engine import Engine

    p, sph, dem = _bed(3, heat, 0, 1)
    p.kgc_solve, p.freq_filt = kgc, freq_filt
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
