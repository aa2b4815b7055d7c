"""Four-Russians products around the shortest K that is cut into slices, both
tile forms, against the oracle."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("k", [15, 16, 17, 80, 81, 96, 97, 112, 113, 128, 129, 192])
def test_short_k(cuda, k, tile):
    for m, n in ((1, 1), (70, 130), (513, 2049)):
        A, B = O.rand_dense(51, 0, m, k), O.rand_dense(51, 1, k, n)
        got = device.matmul(to_dev(A), to_dev(B), m, k, n, _lib.tune(_lib.GEMM_M4RI, 0, tile))
        assert np.array_equal(to_host(got), O.matmul(A, B, m, k, n))
