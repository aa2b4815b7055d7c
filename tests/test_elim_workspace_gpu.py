"""Eliminations on a workspace that is only 8-byte aligned (AUTO and the
Four-Russians form), and Four-Russians on one with room for the panels but not
for the windows.  Against the plain form."""
import pytest

from mex_linear_algebra_b200 import _lib, device

pytestmark = pytest.mark.gpu


def _shifted(nbytes):
    import torch
    return torch.empty(max(nbytes, 1) + 8, dtype=torch.uint8, device="cuda")[8:]


@pytest.mark.parametrize("form", ["M4RI", "AUTO"])
@pytest.mark.parametrize("rref", [False, True])
@pytest.mark.parametrize("m,n,rank", [(60, 150, 50), (300, 700, 280), (700, 500, 333), (1500, 2100, 1400)])
@pytest.mark.parametrize("short", [False, True])
def test_elimination_on_other_workspaces(cuda, form, rref, m, n, rank, short):
    import torch
    if short and form == "AUTO":
        pytest.skip("AUTO wants the size mela_elim_workspace_size names")
    L = _lib.lib()
    left, right = device.rand_dense(23, 0, m, rank), device.rand_dense(23, 1, rank, n)
    A = device.matmul(left, right, m, rank, n)
    wsb = int(L.mela_elim_workspace_size(m, n))
    s = torch.cuda.current_stream().cuda_stream
    got = []
    # short: room for the panels (rows' state and words, 64 reduced rows), not
    # for the windows' byte operands
    small = 64 * ((n + 63) // 64) * 8 + 24 * m + 8192
    for v, ws, nb in ((_lib.ELIM_PLAIN, torch.empty(wsb, dtype=torch.uint8, device="cuda"), wsb),
                      (getattr(_lib, "ELIM_" + form), torch.empty(wsb, dtype=torch.uint8, device="cuda") if short
                       else _shifted(wsb), small if short else wsb)):
        W = A.clone()
        r = torch.zeros(1, dtype=torch.int64, device="cuda")
        piv = torch.zeros(min(m, n), dtype=torch.int64, device="cuda")
        prow = torch.zeros(min(m, n), dtype=torch.int64, device="cuda")
        fn = L.mela_dev_rref if rref else L.mela_dev_rank
        _lib.check(fn(v, W.data_ptr(), W.shape[1], m, n, r.data_ptr(), piv.data_ptr(), prow.data_ptr(), ws.data_ptr(),
                      nb, s))
        k = int(r.item())
        got.append((k, piv[:k].tolist(), W[prow[:k]] if rref else None))
    assert got[0][:2] == got[1][:2]
    assert not rref or torch.equal(got[0][2], got[1][2])
