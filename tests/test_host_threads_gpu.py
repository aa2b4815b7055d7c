"""Page-locked memory of the host entry points: short-lived threads share it (a
set of staging slots and the result words are used again, not made and left
behind by every thread), and results in pieces through shared slots are right
from several threads at once and at the sizes where the copying changes hands
(8 MiB)."""
import os
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rss_mb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE") >> 20


def _product(seed, m, k, n):
    from mex_linear_algebra_b200 import mela
    rng = np.random.default_rng(seed)
    A = np.asfortranarray(rng.integers(0, 2, (m, k)).astype(np.bool_))
    B = np.asfortranarray(rng.integers(0, 2, (k, n)).astype(np.bool_))
    want = (A.astype(np.float32) @ B.astype(np.float32)).astype(np.int32) & 1
    return A, B, want != 0, mela.mela_matmul_gf2


def _in_thread(f):
    bad = []

    def body():
        try:
            f()
        except BaseException as e:
            bad.append(e)
    t = threading.Thread(target=body)
    t.start()
    t.join()
    assert not bad, bad


def test_short_lived_threads_share_the_slots(cuda):
    A, B, want, mul = _product(1, 700, 300, 700)  # a result of 490 KB

    def call():
        for _ in range(3):
            assert np.array_equal(mul(A, B), want)
    for _ in range(3):
        _in_thread(call)
    before = _rss_mb()
    for _ in range(12):
        _in_thread(call)
    assert _rss_mb() - before < 48  # 24 MB of slots a thread would be 288


def test_concurrent_results_in_pieces(cuda):
    cases = [_product(10 + i, 1500 + 400 * i, 200 + 30 * i, 1300) for i in range(8)]
    bad = []

    def work(c):
        A, B, want, mul = c
        try:
            for _ in range(4):
                assert np.array_equal(mul(A, B), want)
        except BaseException as e:
            bad.append(e)
    threads = [threading.Thread(target=work, args=(c,)) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("m,n", [(4096, 2047), (2048, 4096), (2897, 2896), (1048577, 8), (64, 4096), (65, 4096),
                                 (1, 262145)])
def test_sizes_where_the_copying_changes(cuda, m, n):
    A, B, want, mul = _product(m + n, m, 70, n)
    for _ in range(3):
        assert np.array_equal(mul(A, B), want)
