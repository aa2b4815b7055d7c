"""Window factorization of the tensor-core elimination at the edges of its
blocking: 32-column half words, 64 candidate rows a round, 320 rows a chunk,
256 columns a window.  Bit-exact against the oracle (rank, pivot columns, RREF
rows, null basis)."""
import numpy as np
import pytest

from mex_linear_algebra_b200 import gen
from test_elim_gpu import check_all

pytestmark = pytest.mark.gpu


def repeated(m, n, seed):
    """The first 70 rows equal: the first round's 64 candidates span one
    dimension, the other pivots come in later rounds."""
    P = gen.dense_packed(seed, 0, m, n)
    P[: min(70, m)] = P[0]
    return P


def late_pivots(m, n, seed):
    """Rows 0..319 are zero in every even column: the even pivot columns of a
    window come from the second chunk, below and between the first chunk's."""
    P = gen.dense_packed(seed, 0, m, n)
    P[: min(320, m)] &= np.uint64(0xAAAAAAAAAAAAAAAA)
    return P


def low_rank(m, n, seed):
    """Rank 40: every later row reduces to zero through the basis tables."""
    import oracle as O
    L, R = gen.dense_packed(seed, 0, m, 40), gen.dense_packed(seed, 1, 40, n)
    return O.matmul(L, R, m, 40, n)


@pytest.mark.parametrize("make", [repeated, late_pivots, low_rank])
@pytest.mark.parametrize("m,n", [(31, 33), (65, 64), (319, 255), (321, 257), (700, 288), (641, 545)])
def test_window_factor_edges(cuda, make, m, n):
    check_all(make(m, n, 1000 * m + n), m, n, "tc")
