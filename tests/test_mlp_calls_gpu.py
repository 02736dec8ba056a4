"""The network entries' workspace: calls of different sizes one after another, on
other streams, from several threads at once and after a failed call give what a
first call gives (bit for bit), and the thread of a failed wait stays usable.
"""
import os
import threading

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from tests.test_mlp_gpu import _case, _dev, _feat_dev, _lib

pytestmark = pytest.mark.gpu

SIZES = [1, 127, 128, 129, 40_000, 300]


def _run(L, n, seed, stream=None):
    import torch

    p, x, t, w = _case(n, seed)
    w[0] = 1.0
    st = (stream or torch.cuda.current_stream()).cuda_stream
    with torch.cuda.stream(stream) if stream else torch.cuda.stream(torch.cuda.current_stream()):
        f, pd = _feat_dev(x), _dev(p, torch.float32)
        td, wd = _dev(t, torch.float32), _dev(w, torch.float32)
        out = torch.empty(n, dtype=torch.float32, device="cuda")
        g = torch.empty(MO.N_PARAM + 2, dtype=torch.float32, device="cuda")
        torch.cuda.current_stream().synchronize()
        assert L.sphdem_mlp_forward(f.data_ptr(), n, pd.data_ptr(), out.data_ptr(), st) == 0
        assert L.sphdem_mlp_grad(f.data_ptr(), td.data_ptr(), wd.data_ptr(), n, pd.data_ptr(), float(w.sum()),
                                 g.data_ptr(), st) == 0
        return out.cpu().numpy(), g.cpu().numpy()


def test_calls_streams_threads_and_failures_agree():
    import torch

    L = _lib()
    first = {}

    def fresh(n):   # a thread of its own: its first call
        first[n] = _run(L, n, 100 + n)

    for n in SIZES:
        th = threading.Thread(target=fresh, args=(n,))
        th.start()
        th.join()
    same = lambda n, r: all(np.array_equal(a, b) for a, b in zip(first[n], r))   # noqa: E731
    for n in SIZES + SIZES[::-1]:
        assert same(n, _run(L, n, 100 + n))
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k, n in enumerate(SIZES):
        assert same(n, _run(L, n, 100 + n, s[k % 2]))
    got = {}
    ts = [threading.Thread(target=lambda n=n: got.__setitem__(n, [_run(L, n, 100 + n) for _ in range(3)]))
          for n in SIZES]
    for th in ts:
        th.start()
    for th in ts:
        th.join()
    assert all(same(n, r) for n in SIZES for r in got[n])
    # a wait that runs out drops the workspace; the next call builds it again
    n = 300
    p, x, _, _ = _case(n, 7)
    f, pd = _feat_dev(x), _dev(p, torch.float32)
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    os.environ["SPHDEM_FAULT_DRILL"] = "mlp_wait"
    try:
        r = L.sphdem_mlp_forward(f.data_ptr(), n, pd.data_ptr(), out.data_ptr(), None)
    finally:
        del os.environ["SPHDEM_FAULT_DRILL"]
    assert r == -6
    assert same(n, _run(L, n, 100 + n))
