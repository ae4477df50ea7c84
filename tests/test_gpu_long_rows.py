"""Plans of the longest row a request may have, whose rounded-up length does not fit an int."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,dim", [("26.3", "the_nether"), ("26.3", "the_end")])
def test_longest_row(version, dim):
    torch = pytest.importorskip("torch")
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, "normal", 0)
    ow = O.World(ge.data_root(), version, dim, "normal")
    n = 2**31 - 9
    x0 = 2**29 - n  # the row ends at the last quart whose block coordinate is an int
    plan = mg.Plan([(w, 77, x0, 5, n, 1, 16), (w, 78, 3, 4, 33, 18, 16)])
    out = torch.full((plan.output_bytes,), 255, dtype=torch.uint8, device="cuda")
    plan.run_dev(out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for at in (-2**29 - x0, -x0 - 50, -x0 + 8388608 - 4096 - 31, n - 101):  # where the block coordinates are ints
        got = out[at:at + 101].cpu().numpy()
        assert np.array_equal(got, ow.quart_grid(77, x0 + at, 5, 101, 1, 16, O.TIE_ENGINE).reshape(-1)), at
    assert np.array_equal(out[n:].cpu().numpy(), ow.quart_grid(78, 3, 4, 33, 18, 16, O.TIE_ENGINE).reshape(-1))
