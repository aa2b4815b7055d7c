"""Pivot search of the blocked eliminations at the edges of its blocking:
32-column half words and 64 candidate rows a round in every form, 320 rows a
chunk and 256 columns a window in the forms by windows (tensor cores and
Four-Russians tables), 512 rows a chunk and 64 columns a panel in the tuned
Four-Russians form (whose update tiles change from 1024 to 256 rows), 1 to 16 lanes a row and up to 512 rows in the single-CTA form.  Bit-exact against the oracle (rank, pivot columns, RREF rows,
null basis)."""
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
    """The first 512 rows are zero in every even column: the even pivot columns
    come from a later chunk, below and between the first chunk's."""
    P = gen.dense_packed(seed, 0, m, n)
    P[: min(512, m)] &= np.uint64(0xAAAAAAAAAAAAAAAA)
    return P


def low_rank(m, n, seed):
    """Rank 40: every later row reduces to zero through the basis tables."""
    import oracle as O
    L, R = gen.dense_packed(seed, 0, m, 40), gen.dense_packed(seed, 1, 40, n)
    return O.matmul(L, R, m, 40, n)


@pytest.mark.parametrize("make", [repeated, late_pivots, low_rank])
@pytest.mark.parametrize("form,m,n", [("tc", 31, 33), ("tc", 65, 64), ("tc", 319, 255), ("tc", 321, 257),
                                      ("tc", 641, 545), ("tc", 900, 288), ("m4ri_k8", 33, 31), ("m4ri_k8", 511, 65),
                                      ("m4ri_k8", 513, 96), ("m4ri_k8", 1100, 161), ("m4ri_k8", 300, 20000),
                                      ("m4ri", 65, 64), ("m4ri", 321, 257), ("m4ri", 641, 545), ("m4ri", 900, 288),
                                      ("fused", 1, 1), ("fused", 33, 31), ("fused", 65, 129), ("fused", 100, 255),
                                      ("fused", 130, 513), ("fused", 511, 320), ("fused", 512, 2047),
                                      ("fused", 513, 65), ("fused", 90, 7000), ("fused", 200, 8000)])
def test_pivot_search_edges(cuda, make, form, m, n):
    check_all(make(m, n, 1000 * m + n), m, n, form)


@pytest.mark.parametrize("form", ["tc", "m4ri"])
@pytest.mark.parametrize("m,n", [(33, 513), (70, 700), (300, 1100)])
def test_rows_that_leave_the_list(cuda, form, m, n):
    """Zero rows, rows that become zero in the first window and rows whose first
    ones come two windows later: the lists, flags and coefficient slots of the
    later windows, up to windows with no row left."""
    P = gen.dense_packed(m + n, 0, m, n)
    P[::5] = 0
    P[1::5] = P[min(2, m - 1)]
    P[3::5, : (n // 64) // 2] = 0
    check_all(P, m, n, form)
    P[:, 4:] = 0  # no pivots past the first window
    check_all(P, m, n, form)


@pytest.mark.parametrize("form", ["tc", "m4ri"])
@pytest.mark.parametrize("m,n", [(300, 5000), (1400, 1500), (129, 4161)])
def test_update_tiles(cuda, form, m, n):
    """The update of the far columns over one, a few and many row tiles per strip:
    fewer tiles than epilogue groups, strips split between CTAs, a last strip of
    one word."""
    P = gen.dense_packed(m, 0, m, n)
    check_all(P, m, n, form)


@pytest.mark.parametrize("m,n,density", [(700, 260, 0.002), (1000, 600, 0.003), (1300, 520, 0.001), (2100, 300, 0.0006)])
def test_chunks_of_nonzero_rows(cuda, m, n, density):
    """Sparse matrices: chunks gathered from several blocks of the row list,
    blocks that do not fit whole, lists that end inside a chunk."""
    check_all(gen.sparse_packed(11, m, m, n, density), m, n, "m4ri")
