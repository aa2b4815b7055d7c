"""Small products straight from MATLAB-layout arrays: tiles of 32 x 32, K up
to 256 bits, both element kinds, and sizes past where the packed forms take over.  Through the gateways, against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _array(rng, m, n, kind):
    if kind == "logical":
        return np.asfortranarray(rng.integers(0, 2, (m, n)).astype(np.bool_))
    return np.asfortranarray(rng.choice(np.array([0.0, 1.0, -1.0, 2.0, 3.9, -3.5, np.nan, np.inf, 2.0**31, 1e300]),
                                        size=(m, n)))


def _bits(a):
    if a.dtype == np.bool_:
        return a
    ok = (a >= -2.0**31) & (a < 2.0**31)
    return (np.trunc(np.where(ok, a, 0.0)).astype(np.int64) & 1).astype(np.bool_)


@pytest.mark.parametrize("kinds", [("logical", "logical"), ("double", "logical"), ("logical", "double"),
                                   ("double", "double")])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (31, 33, 32), (33, 255, 31), (32, 256, 33), (65, 257, 64), (7, 1100, 90),
                                   (100, 120, 80), (200, 200, 200), (4096, 3, 40), (4097, 3, 40), (512, 256, 512), (300, 200, 300)])
def test_small_products(cuda, kinds, m, k, n):
    from mex_linear_algebra_b200 import mela
    rng = np.random.default_rng(m * 1000 + k + n)
    A, B = _array(rng, m, k, kinds[0]), _array(rng, k, n, kinds[1])
    want = (_bits(A).astype(np.int64) @ _bits(B).astype(np.int64)) & 1
    assert np.array_equal(mela.mela_matmul_gf2(A, B), want != 0)
    assert np.array_equal(mela.mela_matmul_m4ri(A, B), want != 0)
