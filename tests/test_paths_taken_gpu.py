"""Which form a call took, where its results alone do not tell: the seven-product
form leaves most of the workspace alone (a quarter of the operands at a time),
and the fixed rule sends small host calls to the single-CTA form."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base,m,k,n,over,seven", [
    ("tc_fp4", 27150, 27145, 27140, False, True), ("tc_fp4", 16384, 74600, 16385, False, True),
    ("tc_fp4", 16385, 20480, 59700, False, True), ("tc", 20001, 20010, 19990, False, True),
    ("tc", 16640, 30000, 16385, False, True), ("tc_fp4", 27264, 27264, 27264, True, False),
    ("tc_fp4", 16384, 20480, 40000, False, False), ("tc", 16383, 30000, 20000, False, False)])
def test_seven_product_form(cuda, base, m, k, n, over, seven):
    import torch
    from mex_linear_algebra_b200 import device
    A, B = device.rand_dense(11, 0, m, k), device.rand_dense(11, 1, k, n)
    ws = torch.full((device.matmul_workspace(base, m, k, n),), 0xA5, dtype=torch.uint8, device="cuda")
    device.matmul(A, B, m, k, n, base, out=A if over else None, workspace=ws)
    tail = ws[ws.numel() // 2:]
    untouched = bool((tail == 0xA5).all())
    assert untouched == seven


@pytest.mark.parametrize("m,n,rank", [(1, 1, 1), (1, 1, 0), (3, 5, 2), (31, 33, 20), (64, 64, 64), (200, 96, 96),
                                      (100, 481, 60), (255, 511, 255), (256, 512, 200), (128, 512, 0), (100, 513, 90)])
def test_small_calls_by_the_fixed_rule(cuda, m, n, rank):
    from mex_linear_algebra_b200 import _lib, costmodel, mela
    rng = np.random.default_rng(m * 1000 + n + rank)
    A = ((rng.integers(0, 2, (m, rank)) @ rng.integers(0, 2, (rank, n))) & 1).astype(np.bool_)
    A = np.asfortranarray(A)
    want_r, want_z = O.rank(O.pack(A), m, n), np.asarray(O.null_logical(A)) != 0
    L = _lib.lib()
    costmodel.install(None)
    try:
        for _ in range(2):
            assert int(mela.mela_rank_gf2(A)) == want_r
            assert L.mela_dispatch_last(None) == _lib.ELIM_FUSED
            assert np.array_equal(np.asarray(mela.mela_null_gf2(A)) != 0, want_z)
            assert L.mela_dispatch_last(None) == _lib.ELIM_FUSED
    finally:
        costmodel.install_default()
