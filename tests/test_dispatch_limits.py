"""AUTO never resolves to a configuration that refuses the request's size: the
choice without the density, over shapes beyond what single launches take.
Host logic, no GPU."""
import ctypes as C

import pytest

from mex_linear_algebra_b200 import _lib, costmodel

GRID_Y = 65535


def _plan(op, m, n, p=0):
    L = _lib.lib()
    q = C.c_int32(0)
    c = L.mela_costmodel_plan(costmodel.OPS[op], m, n, p, C.byref(q))
    return costmodel.CONFIG_NAMES[op][c] if c >= 0 else None


@pytest.mark.parametrize("m", [128 * GRID_Y, 128 * GRID_Y + 1, 17 << 20, 70 << 20])
@pytest.mark.parametrize("k,n", [(1, 1), (1, 64), (1, 1000), (64, 1), (100, 100)])
def test_tall_products(m, k, n):
    name = _plan("matmul", m, k, n)
    if m > 128 * GRID_Y:
        assert name != "plain"
    if m > 512 * GRID_Y:
        assert not name.startswith("m4ri")


@pytest.mark.parametrize("op", ["rank", "null"])
@pytest.mark.parametrize("m,n", [(70 << 20, 1), (70 << 20, 20), (1 << 30, 64), (17 << 20, 200), (100, 1 << 21),
                                 (3, 1 << 30)])
def test_long_eliminations(op, m, n):
    name = _plan(op, m, n)
    if name is None:
        return
    if n > 64 * 25600:
        assert name != "plain"
    if name.startswith("m4ri"):
        rows = 256 if "rt256" in name else 4096 if "rt4096" in name else 1024
        assert m <= rows * GRID_Y
