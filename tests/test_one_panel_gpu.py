"""Four-Russians and window eliminations of one to five words of columns, where the RREF
goes by panels up to one word: against the oracle."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["M4RI", "M4RI_K4", "TC"])
@pytest.mark.parametrize("m", [1, 2, 63, 300, 1025, 3000])
@pytest.mark.parametrize("n", [1, 3, 63, 64, 65, 128, 256, 257])
def test_few_columns(cuda, form, m, n):
    import torch
    L = _lib.lib()
    rng = np.random.default_rng(m * 1000 + n)
    for density in (0.5, 0.02, 0.0):
        P = O.pack(rng.random((m, n)) < density)
        R, want = O.rref(P, m, n)
        for rref in (False, True):
            W = to_dev(P.copy())
            wsb = int(L.mela_elim_workspace_size(m, n))
            ws = torch.full((wsb,), 0xEE, dtype=torch.uint8, device="cuda")
            r, piv, prow = (torch.full((k,), -7, dtype=torch.int64, device="cuda") for k in (1, min(m, n), min(m, n)))
            fn = L.mela_dev_rref if rref else L.mela_dev_rank
            _lib.check(fn(getattr(_lib, "ELIM_" + form), W.data_ptr(), W.shape[1], m, n, r.data_ptr(), piv.data_ptr(),
                          prow.data_ptr(), ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream))
            k = int(r.item())
            assert piv[:k].tolist() == list(want)
            if rref:
                assert np.array_equal(to_host(W[prow[:k]]), R[:k])
                assert int((W != 0).any(dim=1).sum()) == k
