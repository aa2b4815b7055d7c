"""The single-CTA form on a matrix of more than 2^31 packed words (16 GiB):
three rows with ones, the last of them past the 2^31st word, in one 64-column
panel (a panel without pivots costs a look at every row, one with pivots an
update of every word)."""
import pytest

pytestmark = pytest.mark.gpu


def test_fused_past_2_31_words(cuda):
    import torch
    from mex_linear_algebra_b200 import _lib
    L = _lib.lib()
    m, n = 131080, 1 << 20
    wc = n // 64
    assert (m - 1) * wc >= 1 << 31
    wsb = int(L.mela_elim_workspace_size(m, n))
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < m * wc * 8 + wsb + (1 << 30):
        pytest.skip("needs about 90 GB of device memory")
    M = torch.zeros((m, wc), dtype=torch.int64, device="cuda")
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    # columns 3 and 70000 | 3, 5 and 9 | 5: pivots 3 and 5
    M[7, 0], M[7, 70000 // 64] = 1 << 3, 1 << (70000 % 64)
    M[1000, 0] = (1 << 3) | (1 << 5) | (1 << 9)
    M[m - 1, 0] = 1 << 5
    M[m - 1, wc - 1] = 1 << 62
    rank = torch.zeros(1, dtype=torch.int64, device="cuda")
    piv = torch.zeros(m, dtype=torch.int64, device="cuda")
    prow = torch.zeros(m, dtype=torch.int64, device="cuda")
    _lib.check(L.mela_dev_rref(_lib.ELIM_FUSED, M.data_ptr(), wc, m, n, rank.data_ptr(), piv.data_ptr(),
                               prow.data_ptr(), ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream))
    del ws
    assert int(rank.item()) == 3
    assert piv[:3].tolist() == [3, 5, 9]
    # row 7: 3, 70000; row m - 1: 5, 64 wc - 2; their sum with row 1000: 9, 70000, 64 wc - 2
    want = {3: [3, 70000], 5: [5, 64 * wc - 2], 9: [9, 70000, 64 * wc - 2]}
    for c, r in zip(piv[:3].tolist(), prow[:3].tolist()):
        words = M[r].nonzero().flatten().tolist()
        got = [64 * w + b for w in words for b in range(64) if (int(M[r, w]) >> b) & 1]
        assert got == want[c], (c, got)
    del M
    torch.cuda.empty_cache()
