"""Set bits past the last column: the single-CTA elimination and the batch
engines take them for no columns (the ones before them worked column by column
and never looked there).  Against the same matrices with those bits clear."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _junk(P, n, rng):
    J = P.copy()
    if n % 64:
        extra = rng.integers(0, 1 << 62, size=P.shape[0], dtype=np.int64).astype(np.uint64) * np.uint64(3)
        J[:, -1] |= extra & ~np.uint64((1 << (n % 64)) - 1)
    return J


@pytest.mark.parametrize("m,n", [(1, 1), (5, 3), (40, 33), (100, 20), (72, 149), (300, 65), (200, 500), (250, 447)])
@pytest.mark.parametrize("rref", [False, True])
def test_single_cta(cuda, m, n, rref):
    import torch
    from gpu_util import to_dev
    from mex_linear_algebra_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(m + n)
    P = O.rand_dense(41, m, m, n)
    out = []
    mn = min(m, n)
    for X in (P, _junk(P, n, rng)):
        M = to_dev(X)
        wsb = int(L.mela_elim_workspace_size(m, n))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        rank = torch.zeros(1, dtype=torch.int64, device="cuda")
        piv = torch.full((mn + 64,), -5, dtype=torch.int64, device="cuda")
        prow = torch.full((mn + 64,), -5, dtype=torch.int64, device="cuda")
        fn = L.mela_dev_rref if rref else L.mela_dev_rank
        _lib.check(fn(_lib.ELIM_FUSED, M.data_ptr(), M.shape[1], m, n, rank.data_ptr(), piv.data_ptr(),
                      prow.data_ptr(), ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream))
        r = int(rank.item())
        assert (piv[mn:] == -5).all() and (prow[mn:] == -5).all()
        out.append((r, piv[:r].tolist(), M[prow[:r]] if rref else None))
    assert out[0][:2] == out[1][:2]
    assert not rref or torch.equal(out[0][2], out[1][2])


@pytest.mark.parametrize("count,lo,hi", [(60, 3, 200), (3000, 16, 64), (40, 200, 300)])
def test_batch(cuda, count, lo, hi):
    import torch
    from mex_linear_algebra_b200 import device as D
    rng = np.random.default_rng(count)
    m = rng.integers(lo, hi, size=count)
    shapes = np.stack([m, (m * rng.uniform(0.7, 2.3, size=count)).astype(np.int64) + 1], axis=1)
    clean = [O.rand_dense(42, i, int(a), int(b)) for i, (a, b) in enumerate(shapes)]
    dirty = [_junk(P, int(b), rng) for P, (a, b) in zip(clean, shapes)]
    plan = D.BatchPlan(shapes)
    got = []
    for mats in (clean, dirty):
        d_in = torch.from_numpy(np.concatenate([P.ravel() for P in mats]).view(np.int64)).cuda()
        ranks, zt = plan.run(d_in)
        got.append((ranks.cpu().numpy(), zt.cpu().numpy().view(np.uint64)))
    assert np.array_equal(got[0][0], got[1][0])
    for i in range(count):
        assert np.array_equal(plan.basis(got[0][1], got[0][0], i), plan.basis(got[1][1], got[1][0], i)), i
    plan.close()
