"""The batch engine for whole CTAs, where a matrix and all of its elimination's
storage fit in shared memory and just past that: every shape on both sides of
the line along several aspect ratios, against the oracle; and plans of small
matrices, which need no scratch."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _shapes():
    out = [(1, 1), (1, 64), (1, 65), (64, 1), (3, 5000), (5000, 3), (2, 129), (129, 2)]
    for ratio, lo, hi, step in ((0.3, 330, 640, 17), (1.0, 250, 420, 11), (2.0, 180, 330, 9), (2.3, 170, 300, 9),
                                (4.0, 90, 230, 9), (12.0, 30, 130, 7)):
        out += [(m, max(1, int(m * ratio))) for m in range(lo, hi, step)]
    return out


@pytest.mark.parametrize("kind", ["dense", "sparse", "low rank"])
def test_both_sides_of_shared_memory(cuda, kind):
    import torch
    from mex_linear_algebra_b200 import device as D
    rng = np.random.default_rng(len(kind))
    mats = []
    for m, n in _shapes():
        if kind == "dense":
            a = rng.integers(0, 2, (m, n))
        elif kind == "sparse":
            a = np.zeros((m, n), dtype=np.int64)
            a[np.arange(m)[:, None], rng.integers(0, n, (m, min(6, n)))] = 1
        else:
            r = max(1, min(m, n) // 3)
            a = (rng.integers(0, 2, (m, r)) @ rng.integers(0, 2, (r, n))) & 1
        mats.append(O.pack(a.astype(np.bool_)))
    want = [(O.rank(P, m, n), O.null_basis_packed(P, m, n)) for P, (m, n) in zip(mats, _shapes())]
    # all in one plan (with scratch), and each in a plan of its own (without, where it fits)
    for groups in ([list(range(len(mats)))], [[i] for i in range(len(mats))]):
        for ids in groups:
            plan = D.BatchPlan(np.array([_shapes()[i] for i in ids], dtype=np.int64), force_class=0)
            d_in = torch.from_numpy(np.concatenate([mats[i].ravel() for i in ids]).view(np.int64)).cuda()
            ranks, zt = plan.run(d_in)
            ranks, zt = ranks.cpu().numpy(), zt.cpu().numpy().view(np.uint64)
            for j, i in enumerate(ids):
                m, n = _shapes()[i]
                assert ranks[j] == want[i][0], (m, n)
                assert np.array_equal(plan.basis(zt, ranks, j), want[i][1]), (m, n)
            plan.close()


@pytest.mark.parametrize("count,lo,hi", [(200, 64, 128), (300, 64, 240), (20, 200, 240)])
def test_plans_of_small_matrices_take_no_scratch(cuda, count, lo, hi):
    import torch
    from mex_linear_algebra_b200 import device as D
    rng = np.random.default_rng(count)
    m = rng.integers(lo, hi, size=count)
    shapes = np.stack([m, 2 * m + rng.integers(0, 1 + m // 4)], axis=1)
    D.BatchPlan(shapes).close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = D.BatchPlan(shapes)
    taken = before - torch.cuda.mem_get_info()[0]
    assert plan.stats()["cta"] == count
    plan.close()
    assert taken <= 4 << 20  # the item list; scratch for 296 CTAs would be 6 to 25 MB
