"""Small rank and null-space calls whose kernel writes the result straight into
page-locked words: columns at and beside word and capacity edges, more and fewer
rows than columns, empty and full bases, repeated calls, and an allocator that
calls back into the library.  Against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _oracle(A):
    return O.rank(O.pack(A), *A.shape), np.asarray(O.null_logical(A)) != 0


@pytest.mark.parametrize("m,n,rank", [(1, 1, 1), (1, 1, 0), (3, 5, 2), (31, 33, 20), (64, 64, 64), (72, 149, 70),
                                      (200, 96, 96), (100, 481, 60), (255, 511, 255), (256, 512, 200), (128, 512, 0),
                                      (100, 513, 90), (512, 130, 128)])
@pytest.mark.parametrize("kind", [np.bool_, np.float64])
def test_small_rank_and_null(cuda, m, n, rank, kind):
    from mex_linear_algebra_b200 import mela
    rng = np.random.default_rng(m * 1000 + n + rank)
    A = ((rng.integers(0, 2, (m, rank)) @ rng.integers(0, 2, (rank, n))) & 1).astype(kind)
    A = np.asfortranarray(A)
    want_r, want_z = _oracle(A != 0)
    for _ in range(2):
        assert int(mela.mela_rank_gf2(A)) == want_r
        assert np.array_equal(np.asarray(mela.mela_null_gf2(A)) != 0, want_z)


def test_allocator_calls_back(cuda):
    """The basis survives another null-space call from inside the allocator."""
    from mex_linear_algebra_b200 import _lib, mela
    rng = np.random.default_rng(5)
    A = np.asfortranarray(rng.integers(0, 2, (60, 140)).astype(np.bool_))
    B = np.asfortranarray(rng.integers(0, 2, (40, 90)).astype(np.bool_))
    box = {}

    def alloc(ctx, rows, cols):
        box["inner"] = np.asarray(mela.mela_null_gf2(B)) != 0
        box["z"] = np.zeros((rows, cols), dtype=np.uint8, order="F")
        return box["z"].ctypes.data
    H = _lib.HostMatrix()
    H.rows, H.cols, H.kind, H.sparse, H.data = 60, 140, _lib.KIND_LOGICAL, 0, A.ctypes.data
    f = C.c_int64(0)
    _lib.check(_lib.lib().mela_null_gf2(C.byref(H), _lib.ALLOC_FN(alloc), None, C.byref(f)))
    assert np.array_equal(box["z"] != 0, _oracle(A)[1])
    assert np.array_equal(box["inner"], _oracle(B)[1])
