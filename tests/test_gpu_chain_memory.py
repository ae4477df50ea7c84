"""Device memory that the candidate-chain rules' grids take: 44 bytes a cell (a record of 40 and its place in the order)."""
import ctypes as C

import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu
USED_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


@pytest.mark.parametrize("version", ["26.1", "26.3"])
def test_scratch(version):
    torch = pytest.importorskip("torch")
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", "normal", 5)
    ow = O.World(ge.data_root(), version, "overworld")
    nx, nz = 1501, 999
    out = torch.empty(nx * nz, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    cu, pool, v = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    for rule in (mg.TIE_GRID_CHAIN, mg.TIE_CHUNK_ORDER):
        torch.cuda.synchronize()
        zero = C.c_uint64(0)
        assert cu.cuMemPoolSetAttribute(pool, USED_HIGH, C.byref(zero)) == 0
        assert cu.cuMemPoolGetAttribute(pool, USED_HIGH, C.byref(v)) == 0
        before = v.value
        w.quart_grid_dev(-700, 31, nx, nz, 16, rule, out.data_ptr(), stream)
        torch.cuda.synchronize()
        assert cu.cuMemPoolGetAttribute(pool, USED_HIGH, C.byref(v)) == 0
        assert v.value - before <= 44 * nx * nz + (1 << 16), rule
    assert np.array_equal(out.cpu().numpy().reshape(nz, nx), ow.chunk_order_grid(5, -700, 31, nx, nz, 16))
