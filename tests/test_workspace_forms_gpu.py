"""Products whose buffers rule a form out: a workspace that is only 8-byte
aligned (AUTO takes a form that allows it, the tensor-core forms refuse it), and
AUTO products written over an operand or beside it in one buffer.  Against the
oracle."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


def _shifted(nbytes):
    import torch
    return torch.empty(max(nbytes, 1) + 8, dtype=torch.uint8, device="cuda")[8:]


@pytest.mark.parametrize("m,k,n", [(100, 120, 80), (64, 2000, 64), (400, 300, 600), (700, 1100, 900),
                                   (1100, 1200, 1300)])
def test_auto_product_on_an_unaligned_workspace(cuda, m, k, n):
    import torch
    A, B = O.rand_dense(21, 0, m, k), O.rand_dense(21, 1, k, n)
    want = O.matmul(A, B, m, k, n)
    a, b = to_dev(A), to_dev(B)
    ws = _shifted(device.matmul_workspace("auto", m, k, n))
    got = device.matmul(a, b, m, k, n, workspace=ws)
    assert np.array_equal(to_host(got), want)
    L, out = _lib.lib(), torch.full_like(got, -1)
    s = torch.cuda.current_stream().cuda_stream
    args = (0, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1])
    _lib.check(L.mela_dev_matmul_prepare(*args, m, k, n, ws.data_ptr(), ws.numel(), s))
    _lib.check(L.mela_dev_matmul_run(*args, out.data_ptr(), out.shape[1], m, k, n, ws.data_ptr(), ws.numel(), s))
    assert torch.equal(out, got)


@pytest.mark.parametrize("n", [64, 200, 300, 512, 1000, 2100])
@pytest.mark.parametrize("over", ["A", "B"])
def test_auto_product_over_an_operand(cuda, n, over):
    A, B = O.rand_dense(22, 0, n, n), O.rand_dense(22, 1, n, n)
    want = O.matmul(A, B, n, n, n)
    a, b = to_dev(A), to_dev(B)
    out = a if over == "A" else b
    device.matmul(a, b, n, n, n, out=out)
    assert np.array_equal(to_host(out), want)


@pytest.mark.parametrize("n", [64, 300, 640])
def test_auto_product_beside_an_operand(cuda, n):
    """A and C as column blocks of one buffer."""
    import torch
    A, B = O.rand_dense(24, 0, n, n), O.rand_dense(24, 1, n, n)
    want = O.matmul(A, B, n, n, n)
    w = A.shape[1]
    buf = torch.full((n, 2 * w), -1, dtype=torch.int64, device="cuda")
    buf[:, :w] = to_dev(A)
    b = to_dev(B)
    L, s = _lib.lib(), torch.cuda.current_stream().cuda_stream
    wsb = device.matmul_workspace("auto", n, n, n)
    ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device="cuda")
    _lib.check(L.mela_dev_matmul(0, buf.data_ptr(), 2 * w, b.data_ptr(), w, buf.data_ptr() + 8 * w, 2 * w, n, n, n,
                                 ws.data_ptr(), wsb, s))
    assert np.array_equal(to_host(buf)[:, w:], want)
    assert np.array_equal(to_host(buf)[:, :w], A)


@pytest.mark.parametrize("form", ["tc", "tc_fp4"])
def test_tensor_core_forms_refuse_an_unaligned_workspace(cuda, form):
    m, k, n = 300, 400, 500
    A, B = device.rand_dense(25, 0, m, k), device.rand_dense(25, 1, k, n)
    with pytest.raises(Exception, match="aligned"):
        device.matmul(A, B, m, k, n, form, workspace=_shifted(device.matmul_workspace(form, m, k, n)))
