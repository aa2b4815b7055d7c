"""Eliminations by windows of matrices with many more rows than columns, where the
rows that complete a window's basis lie far down the list or are missing: against
the oracle; and the time of a rank that used to walk every row for its last
columns."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


def _run(form, M, m, n, rref):
    import torch
    L = _lib.lib()
    W = M.clone()
    wsb = int(L.mela_elim_workspace_size(m, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    r = torch.zeros(1, dtype=torch.int64, device="cuda")
    piv = torch.zeros(min(m, n), dtype=torch.int64, device="cuda")
    prow = torch.zeros(min(m, n), dtype=torch.int64, device="cuda")
    fn = L.mela_dev_rref if rref else L.mela_dev_rank
    _lib.check(fn(form, W.data_ptr(), W.shape[1], m, n, r.data_ptr(), piv.data_ptr(), prow.data_ptr(), ws.data_ptr(),
                  wsb, torch.cuda.current_stream().cuda_stream))
    k = int(r.item())
    return k, piv[:k].tolist(), to_host(W[prow[:k]]) if rref else None, W


def _check(form, P, m, n):
    M = to_dev(P)
    want_rows, want_piv = O.rref(P, m, n)[:2]
    for rref in (False, True):
        k, piv, rows, W = _run(form, M, m, n, rref)
        assert piv == list(want_piv), (form, rref)
        if rref:
            assert np.array_equal(rows, want_rows[:k])
            assert int((W != 0).any(dim=1).sum()) == k  # the other rows are zero


@pytest.mark.parametrize("form", ["TC", "M4RI"])
@pytest.mark.parametrize("m,n,density", [(2000, 1, 0.01), (3000, 2, 0.001), (4000, 64, 0.002), (3000, 257, 0.004),
                                         (5000, 700, 0.002), (1500, 300, 0.5), (641, 320, 0.02)])
def test_windows(cuda, form, m, n, density):
    rng = np.random.default_rng(m + n)
    a = rng.random((m, n)) < density
    _check(getattr(_lib, "ELIM_" + form), O.pack(a), m, n)
    # the same with the rows that complete the basis at the very end, most of the list empty
    b = np.zeros_like(a)
    b[:40] = rng.random((40, n)) < 0.5
    b[m // 2] = True
    q = min(n, 60)
    b[m - q:, :q] = np.triu(np.ones((q, q), dtype=bool))
    _check(getattr(_lib, "ELIM_" + form), O.pack(b), m, n)


def test_rank_of_a_tall_sparse_matrix_in_time(cuda):
    import torch
    L, m, n = _lib.lib(), 1000000, 64
    M = torch.empty((m, 1), dtype=torch.int64, device="cuda")
    _lib.check(L.mela_dev_rand_bernoulli(3, 1, m, n, 0.001, M.data_ptr(), 1, 0))
    W = M.clone()
    wsb = int(L.mela_elim_workspace_size(m, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    r, piv, prow = (torch.zeros(k, dtype=torch.int64, device="cuda") for k in (1, n, n))
    best = 1e9
    for _ in range(6):
        W.copy_(M)
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        _lib.check(L.mela_dev_rank(_lib.ELIM_TC, W.data_ptr(), 1, m, n, r.data_ptr(), piv.data_ptr(), prow.data_ptr(),
                                   ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream))
        e1.record()
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    assert int(r.item()) == n
    assert best < 1.0  # ms: 0.17 measured, 3.5 when every row is walked
