"""The single-CTA elimination of matrices with more than 512 rows, on both sides of
the line between its two engines.  Against the oracle."""
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


@pytest.mark.parametrize("m,n", [(513, 1), (513, 24), (513, 25), (1024, 24), (1025, 25), (1025, 130), (3000, 2),
                                 (2000, 480), (2000, 481), (20000, 3)])
@pytest.mark.parametrize("density", [0.5, 0.01])
def test_single_cta(cuda, m, n, density):
    rng = np.random.default_rng(m + n)
    _check(_lib.ELIM_FUSED, O.pack(rng.random((m, n)) < density), m, n)
