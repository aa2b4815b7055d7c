"""Results of every size the host entry points bring down: through the
thread's page-locked words (up to 256 KiB), by one direct copy, and in pieces
through the staging slots (1 MiB and larger: ragged last pieces, more pieces
than slots), from several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(seed, m, n, k=70):
    from mex_linear_algebra_b200 import mela
    rng = np.random.default_rng(seed)
    A = np.asfortranarray(rng.integers(0, 2, (m, k)).astype(np.bool_))
    B = np.asfortranarray(rng.integers(0, 2, (k, n)).astype(np.bool_))
    want = (A.astype(np.float32) @ B.astype(np.float32)).astype(np.int32) & 1
    assert np.array_equal(mela.mela_matmul_gf2(A, B), want != 0)


@pytest.mark.parametrize("m,n", [(512, 512), (513, 512), (1023, 1025), (1024, 1024), (1025, 1024), (2731, 1537),
                                 (4001, 2500), (6001, 5999)])
def test_result_sizes(cuda, m, n):
    _check(m + n, m, n)


def test_results_from_threads(cuda):
    bad = []

    def work(i):
        try:
            for r in range(3):
                _check(10 * i + r, 1500 + 100 * i, 1400)
                _check(10 * i + r, 60 + i, 50)
        except BaseException as e:  # reported by the main thread
            bad.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
