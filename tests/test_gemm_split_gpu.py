"""Products with K in slices (Four-Russians, and single-CTA tensor cores): slice counts from one to the last
partial slice, B addressable by TMA or not, into a result buffer that held
other bits and whose padding must stay."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (100, 64, 80), (100, 65, 80), (513, 130, 2100), (70, 1000, 129),
                                   (600, 2000, 65), (2000, 9501, 100)])
def test_k_slices(cuda, m, k, n, tile):
    import torch
    A, B = O.rand_dense(3, 0, m, k), O.rand_dense(3, 1, k, n)
    want = O.matmul(A, B, m, k, n)
    wn = (n + 63) // 64
    for pad in (wn % 2, 1 - wn % 2):  # an even and an odd row pitch of B
        Bp = np.zeros((k, wn + pad), dtype=np.uint64)
        Bp[:, :wn] = B
        out = torch.full((m, wn + 1), -1, dtype=torch.int64, device="cuda")
        device.matmul(to_dev(A), to_dev(Bp), m, k, n, _lib.tune(_lib.GEMM_M4RI, 0, tile), out=out)
        got = to_host(out)
        assert np.array_equal(got[:, :wn], want)
        assert (out[:, wn:] == -1).all()


@pytest.mark.parametrize("base", [_lib.GEMM_TC, _lib.GEMM_TC_FP4])
@pytest.mark.parametrize("m,k,n", [(1, 4097, 1), (100, 3841, 300), (130, 2049, 257), (300, 20001, 260),
                                   (700, 4200, 1300)])
def test_tensor_core_k_slices(cuda, base, m, k, n):
    import torch
    A, B = O.rand_dense(5, 0, m, k), O.rand_dense(5, 1, k, n)
    want = O.matmul(A, B, m, k, n)
    wn = (n + 63) // 64
    out = torch.full((m, wn + 1), -1, dtype=torch.int64, device="cuda")
    device.matmul(to_dev(A), to_dev(B), m, k, n, _lib.tune(base, 0, 1), out=out)
    assert np.array_equal(to_host(out)[:, :wn], want)
    assert (out[:, wn:] == -1).all()
