"""Operand expansion of the tensor-core products: rows on and off 16-byte
boundaries (odd pitches, a base one word into its buffer), K and columns at and
beside the 256-bit tiles, more pieces than one pass of the grid -- against the
table-driven product, which reads the packed words themselves."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["tc", "tc_fp4"])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (130, 255, 257), (256, 256, 256), (300, 513, 767), (2050, 4096, 1024),
                                   (9000, 2111, 3000)])
@pytest.mark.parametrize("pad,offset", [(0, 0), (1, 0), (2, 1)])
def test_operand_alignment(cuda, variant, m, k, n, pad, offset):
    import torch
    from mex_linear_algebra_b200 import device

    def operand(rows, cols, stream_id):
        ld = device.words(cols) + pad
        x = torch.full((rows * ld + offset,), -1, dtype=torch.int64, device="cuda")[offset:].view(rows, ld)
        x[:, :device.words(cols)] = device.rand_dense(21, stream_id, rows, cols)
        return x
    A, B = operand(m, k, 0), operand(k, n, 1)
    got = device.matmul(A, B, m, k, n, variant)
    assert torch.equal(got, device.matmul(A, B, m, k, n, "m4ri"))
