"""Four-Russians products written over an operand, where every block of the
result is written by the one CTA that reads those words: over A up to 2048
columns, over B up to 512 rows.  K long enough for slices, both tile forms."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("m,k,n,over", [(512, 512, 512, "A"), (100, 65, 65, "A"), (2000, 2048, 2048, "A"),
                                        (513, 300, 260, "A"), (512, 512, 512, "B"), (65, 130, 100, "B"),
                                        (500, 512, 3000, "B")])
def test_result_over_an_operand(cuda, m, k, n, over, tile):
    A, B = O.rand_dense(7, 0, m, k), O.rand_dense(7, 1, k, n)
    want = O.matmul(A, B, m, k, n)
    wn = (n + 63) // 64
    a, b = to_dev(A), to_dev(B)
    buf = a if over == "A" else b
    assert buf.shape[1] >= wn and buf.shape[0] >= m
    out = buf[:m]
    device.matmul(a, b, m, k, n, _lib.tune(_lib.GEMM_M4RI, 0, tile), out=out)
    assert np.array_equal(to_host(out)[:, :wn], want)
