"""The network entries at the largest row count they take, 2^31 - 128: the row of a CTA's next tile lies past 2^31
there.  Needs 90 GB of device memory (the features alone are 69 GB).

Bar: a row's output depends on that row alone, so the outputs of the first and last rows equal those of a call on
just these rows bit for bit.  All weights but theirs are zero, so the gradient is theirs: the bar of the gradient
against the oracle elsewhere (5e-3 per parameter block, loss 1e-4, weight sum 1e-6).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from tests.test_mlp_gpu import _case, _dev, _feat_dev, _lib, _rel

pytestmark = pytest.mark.gpu

ROWS = 2**31 - 128
EDGE = 50_000   # rows in use at each end


def test_largest_row_count():
    import torch

    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 90 GB of free device memory")
    L = _lib()
    p, x, t, w = _case(2 * EDGE, 3)
    feat, target, weight, params = _feat_dev(x), _dev(t, torch.float32), _dev(w, torch.float32), _dev(p, torch.float32)
    st = torch.cuda.current_stream().cuda_stream
    out = torch.empty(2 * EDGE, dtype=torch.float32, device="cuda")
    assert L.sphdem_mlp_forward(feat.data_ptr(), 2 * EDGE, params.data_ptr(), out.data_ptr(), st) == 0
    try:
        big = torch.zeros((ROWS, MO.N_IN), dtype=torch.bfloat16, device="cuda")
        big[:EDGE], big[-EDGE:] = feat[:EDGE], feat[EDGE:]
        y = torch.empty(ROWS, dtype=torch.float32, device="cuda")
        assert L.sphdem_mlp_forward(big.data_ptr(), ROWS, params.data_ptr(), y.data_ptr(), st) == 0
        assert torch.equal(y[:EDGE], out[:EDGE]) and torch.equal(y[-EDGE:], out[EDGE:])
        wb = torch.zeros(ROWS, dtype=torch.float32, device="cuda")
        y.zero_()   # the targets
        for a, v in ((y, target), (wb, weight)):
            a[:EDGE], a[-EDGE:] = v[:EDGE], v[EDGE:]
        g = torch.empty(MO.N_PARAM + 2, dtype=torch.float32, device="cuda")
        assert L.sphdem_mlp_grad(big.data_ptr(), y.data_ptr(), wb.data_ptr(), ROWS, params.data_ptr(), float(w.sum()),
                                 g.data_ptr(), st) == 0
        g = g.cpu().numpy().astype(np.float64)
    finally:
        big = y = wb = None
        torch.cuda.empty_cache()
    go, loss, wsum = MO.grad(p, x, t, w, float(w.sum()))
    cuts = [MO.OFF_W1, MO.OFF_B1, MO.OFF_W2, MO.OFF_B2, MO.OFF_W3, MO.OFF_B3, MO.N_PARAM]
    assert all(_rel(g[a:b], go[a:b]) <= 5e-3 for a, b in zip(cuts, cuts[1:]))
    assert abs(g[MO.N_PARAM] - loss) <= 1e-4 * loss
    assert abs(g[MO.N_PARAM + 1] - wsum) <= 1e-6 * wsum
