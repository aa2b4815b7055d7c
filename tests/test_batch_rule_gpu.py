"""The size rule of batch plans: which engine takes small matrices depends on how
many there are (warps where they save more slot time than a late one costs);
the results do not.  Against the oracle and against every matrix on CTAs."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,lo,hi,engine", [(40, 8, 192, "cta"), (6000, 8, 64, "warp"), (3000, 150, 200, None),
                                                (5000, 16, 128, "warp"), (700, 30, 260, None), (1, 1, 2, "warp")])
def test_engine_by_count(cuda, count, lo, hi, engine):
    import torch
    from mex_linear_algebra_b200 import device as D
    rng = np.random.default_rng(count + lo)
    m = rng.integers(lo, hi, size=count)
    n = (m * rng.uniform(1.0, 2.3, size=count)).astype(np.int64) + 1
    shapes = np.stack([m, n], axis=1)
    plan, ctas = D.BatchPlan(shapes), D.BatchPlan(shapes, force_class=0)
    st = plan.stats()
    assert st["group128"] == 0
    if engine is not None:
        assert st[engine] == count, st
    d_in = torch.zeros(plan.in_words, dtype=torch.int64, device="cuda")
    host = np.zeros(plan.in_words, dtype=np.uint64)
    for i in range(count):
        P = O.pack(rng.integers(0, 2, (int(m[i]), int(n[i])), dtype=np.uint8).astype(np.bool_))
        o = int(plan.in_offsets[i])
        host[o:o + P.size] = P.ravel()
    d_in.copy_(torch.from_numpy(host.view(np.int64)))
    ra, za = plan.run(d_in)
    rb, zb = ctas.run(d_in)
    ra, rb = ra.cpu().numpy(), rb.cpu().numpy()
    za, zb = za.cpu().numpy().view(np.uint64), zb.cpu().numpy().view(np.uint64)
    assert np.array_equal(ra, rb)
    for i in range(count):
        assert np.array_equal(plan.basis(za, ra, i), ctas.basis(zb, rb, i)), i
    for i in range(0, count, max(1, count // 20)):
        o, wc = int(plan.in_offsets[i]), int(plan.wc[i])
        P = host[o:o + int(m[i]) * wc].reshape(int(m[i]), wc)
        assert ra[i] == O.rank(P, int(m[i]), int(n[i]))
        assert np.array_equal(plan.basis(za, ra, i), O.null_basis_packed(P, int(m[i]), int(n[i])))
    plan.close()
    ctas.close()
