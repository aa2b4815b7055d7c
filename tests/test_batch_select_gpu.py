"""The batch engine's pivot selection at the edges of its register widths (64,
128, 192, 256 and 384 candidate rows), with pivots in either half of the panel's
word only, and the two-word update over odd and even row widths.  Against the
oracle."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_host
from mex_linear_algebra_b200 import gen

pytestmark = pytest.mark.gpu


def _matrix(m, n, cand, mask, seed):
    """`cand` rows of the first panel random under `mask`, the others zero there."""
    P = gen.dense_packed(seed, 0, m, n)
    P[:, 0] &= np.uint64(mask)
    P[cand:, 0] = 0
    P[:cand:2, 0] |= P[1:cand:2, 0][0] if cand > 1 else P[0, 0]
    return P


def test_selection_widths(cuda):
    import torch
    from mex_linear_algebra_b200 import device as D
    full, low, high = 0xFFFFFFFFFFFFFFFF, 0x00000000FFFFFFFF, 0xFFFFFFFF00000000
    mats = []
    for i, (cand, mask) in enumerate([(1, full), (2, low), (63, high), (64, full), (65, full), (128, low), (129, full),
                                      (192, high), (193, full), (256, full), (257, low), (384, full), (385, full)]):
        for n in (260 + 64 * (i % 3), 700):
            m = max(cand + 7, 250)
            mats.append((m, n, _matrix(m, n, cand, mask, 100 * i + n)))
    plan = D.BatchPlan([(m, n) for (m, n, _) in mats], force_class=0)
    buf = np.zeros(plan.in_words, dtype=np.uint64)
    for i, (m, n, P) in enumerate(mats):
        o = int(plan.in_offsets[i])
        buf[o:o + P.size] = P.ravel()
    ranks, zt = plan.run(torch.from_numpy(buf.view(np.int64)).cuda())
    rk, z = to_host(ranks), to_host(zt)
    for i, (m, n, P) in enumerate(mats):
        assert rk[i] == len(O.rref(P, m, n)[1])
        assert np.array_equal(plan.basis(z, rk, i), O.null_basis_packed(P, m, n)), (m, n)
    plan.close()
