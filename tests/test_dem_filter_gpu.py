"""The DEM filter of Wendland C2 where its lists fill: spheres with more SPH neighbours than the coupling's list holds
(256), and with more than the filter's own (512), which are scanned again.

Bars as in test_set_sizes_gpu.py: FP64 build vs the FP64 oracle 1e-9 per field, FP32 vs FP64 build 1e-5 for state and
1e-4 for rate fields after 2 steps.
"""
import numpy as np
import pytest

from fluidized_bed_master_b200.beds import box_bed
from tests.test_set_sizes_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide,most", [(1.6, 257), (2.2, 520)])
def test_full_lists(wide, most):
    p, sph, dem = box_bed(n_fluid=5_001, n_dem=101, dem_height=0.012, lx=0.02, seed=23)
    p.h_over_dx *= wide
    sph["h"] = sph["h"] * wide
    dem["h"] = dem["h"] * wide
    d2 = sum((sph[c][None] - dem[c][:, None]) ** 2 for c in "xyz")
    n = (d2 < (p.kappa * dem["h"][:, None]) ** 2).sum(1)
    assert n.max() > most
    _compare(p, sph, dem)
