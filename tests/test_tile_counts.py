"""Tiles of a grid: rows and columns up to the largest int."""
import ctypes as C

import pytest

import __graft_entry__ as ge


@pytest.fixture(scope="module")
def ow_tiles():
    ge._build_module().build()
    f = C.CDLL(ge.package().LIB_PATH)._ZN2mg8ow_tilesEii  # long long mg::ow_tiles(int, int)
    f.restype, f.argtypes = C.c_longlong, [C.c_int, C.c_int]
    return f


@pytest.mark.parametrize("n", [1, 15, 16, 17, 2**30 + 1, 2**31 - 17, 2**31 - 16, 2**31 - 15, 2**31 - 1])
def test_overworld_tiles(ow_tiles, n):
    assert ow_tiles(n, 1) == ow_tiles(1, n) == (n + 15) // 16
    assert ow_tiles(n, 17) == 2 * ((n + 15) // 16)
