"""Large products by seven products of half-size blocks: against the two-call
form (prepare, run), which multiplies the whole matrices, at the smallest sizes
of the rule, ragged in every dimension, with row pitches wider than the matrix
and with the result written over an operand (which takes the whole form)."""
import pytest

pytestmark = pytest.mark.gpu


def _whole(L, check, v, A, B, C, m, k, n, ws, s):
    a = (v, A.data_ptr(), A.shape[1], B.data_ptr(), B.shape[1])
    check(L.mela_dev_matmul_prepare(*a, m, k, n, ws.data_ptr(), ws.numel(), s))
    check(L.mela_dev_matmul_run(*a, C.data_ptr(), C.shape[1], m, k, n, ws.data_ptr(), ws.numel(), s))


@pytest.mark.parametrize("base,m,k,n,pad", [
    ("tc_fp4", 27150, 27145, 27140, 0),   # just past the smallest volume
    ("tc_fp4", 16384, 74600, 16385, 3),   # the smallest rows, a long K
    ("tc_fp4", 16385, 20480, 59700, 1),   # the smallest K, a wide result
    ("tc", 20001, 20010, 19990, 2),
    ("tc", 16640, 30000, 16385, 0),
])
def test_seven_products(cuda, base, m, k, n, pad):
    import torch
    from mex_linear_algebra_b200 import _lib, device
    L, v = _lib.lib(), _lib.GEMM_VARIANTS[base]
    wk, wn = device.words(k), device.words(n)
    A = device.rand_dense(11, 0, m, k, ld=wk + pad)
    B = device.rand_dense(11, 1, k, n, ld=wn + pad)
    want = torch.full((m, wn), -1, dtype=A.dtype, device="cuda")
    got = torch.full((m, wn + pad), -1, dtype=A.dtype, device="cuda")
    ws = torch.empty(device.matmul_workspace(base, m, k, n), dtype=torch.uint8, device="cuda")
    _whole(L, _lib.check, v, A, B, want, m, k, n, ws, torch.cuda.current_stream().cuda_stream)
    device.matmul(A, B, m, k, n, base, out=got, workspace=ws)
    assert torch.equal(got[:, :wn], want)
    assert pad == 0 or bool((got[:, wn:] == -1).all())  # nothing past the result's words
    assert L.mela_device_error_flags(None, 0) == 0


def test_result_over_an_operand(cuda):
    import torch
    from mex_linear_algebra_b200 import device
    n = 27264
    A = device.rand_dense(12, 0, n, n)
    B = device.rand_dense(12, 1, n, n)
    want = device.matmul(A, B, n, n, n, "tc_fp4")
    device.matmul(A, B, n, n, n, "tc_fp4", out=A)
    assert torch.equal(A, want)
