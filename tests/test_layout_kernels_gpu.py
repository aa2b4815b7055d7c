"""Packing, unpacking and the null-space basis at the edges of their tiles
(128 rows, 64-column words, 16-byte output pieces), from bases at every
alignment.  Exact against numpy and the oracle."""
import numpy as np
import pytest

import oracle as O
from gpu_util import to_dev, to_host
from mex_linear_algebra_b200 import _lib, device, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (3, 65), (127, 64), (128, 63), (129, 257), (131, 16), (260, 300), (513, 130), (256, 70)])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_logical_any_alignment(cuda, m, n, shift):
    import torch
    rng = np.random.default_rng(1000 * m + n)
    a = rng.choice(np.array([0, 1, 2, 127, 128, 255], np.uint8), size=(n, m))  # column j is row j here
    buf = torch.zeros(m * n + 16, dtype=torch.uint8, device="cuda")
    buf[shift:shift + m * n] = torch.from_numpy(a.ravel()).cuda()
    ld = (n + 63) // 64 + 1
    P = device.pack(buf[shift:shift + m * n], m, n, ld=ld)
    want = O.pack(np.asfortranarray(a.T != 0), ld)
    assert np.array_equal(to_host(P), want)
    # back, into a window of a larger buffer whose other bytes stay
    out = torch.full((m * n + 16,), 7, dtype=torch.uint8, device="cuda")
    device.unpack(P, m, n, out=out[shift:shift + m * n])
    got = out.cpu().numpy()
    assert np.array_equal(got[shift:shift + m * n], (a.ravel() != 0).astype(np.uint8))
    assert (got[:shift] == 7).all() and (got[shift + m * n:] == 7).all()
    # packed rows to row-major bytes
    rows = torch.full((m * n + 16,), 7, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().mela_dev_unpack_rows(P.data_ptr(), ld, m, n, rows.data_ptr() + shift,
                                               torch.cuda.current_stream().cuda_stream))
    got = rows.cpu().numpy()
    assert np.array_equal(got[shift:shift + m * n].reshape(m, n), (a.T != 0).astype(np.uint8))
    assert (got[:shift] == 7).all() and (got[shift + m * n:] == 7).all()


@pytest.mark.parametrize("m,n", [(1, 17), (31, 64), (33, 130), (70, 300)])
def test_pack_doubles(cuda, m, n):
    import torch
    rng = np.random.default_rng(m + n)
    a = rng.choice(np.array([0.0, 1.0, -1.0, 2.0, 3.9, -3.5, np.nan, np.inf, -np.inf, 2.0**31, -2.0**31, 1e300]),
                   size=(m, n))
    P = device.pack(torch.from_numpy(a.T.copy()).cuda().reshape(-1), m, n)
    assert np.array_equal(to_host(P), O.pack(np.asfortranarray(a)))


@pytest.mark.parametrize("m,n,r", [(1, 1, 0), (1, 200, 1), (64, 64, 63), (65, 129, 64), (200, 257, 130), (300, 320, 256),
                                   (520, 2100, 513)])
def test_null_basis_edges(cuda, m, n, r):
    """Ranks at word edges; pivots packed at the front, and interleaved with
    free columns (every third column a copy of the one before)."""
    import torch
    L = _lib.lib()
    for spread in (False, True):
        bits = O.unpack(O.matmul(gen.dense_packed(7, 0, m, max(r, 1)), gen.dense_packed(7, 1, max(r, 1), n), m,
                                 max(r, 1), n), m, n).copy()
        if r == 0:
            bits[:] = False
        if spread and n > 3:
            bits[:, 2::3] = bits[:, 1::3][:, :bits[:, 2::3].shape[1]]
        P = O.pack(np.asfortranarray(bits))
        R, piv = O.rref(P, m, n)
        k, f = len(piv), n - len(piv)
        dR = to_dev(R)
        dpiv = torch.from_numpy(np.concatenate([piv, [0]])).cuda()
        dprow = torch.arange(max(k, 1), dtype=torch.int64, device="cuda")
        ldz = (n + 63) // 64 + 1
        Zt = torch.full((f + 1, ldz), -1, dtype=torch.int64, device="cuda")
        wsb = L.mela_null_workspace_size(n, k)
        ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device="cuda")
        _lib.check(L.mela_dev_null_basis(dR.data_ptr(), dR.shape[1], m, n, k, dpiv.data_ptr(), dprow.data_ptr(),
                                         Zt.data_ptr(), ldz, ws.data_ptr(), wsb,
                                         torch.cuda.current_stream().cuda_stream))
        got = to_host(Zt)
        assert np.array_equal(got[:f, :-1], O.null_basis_packed(P, m, n))
        assert (Zt[f:] == -1).all() and (Zt[:, -1] == -1).all()


def test_null_workspace_covers_smaller_ranks(cuda):
    """A workspace sized for a rank serves every smaller rank."""
    L = _lib.lib()
    for n in (1, 64, 200, 1000, 4097):
        sizes = [L.mela_null_workspace_size(n, r) for r in range(0, n + 1, max(1, n // 50))]
        assert sizes == sorted(sizes)
