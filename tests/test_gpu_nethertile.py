"""The batch's Nether tiles (32 x 32 cells from tables of lattice nodes) against the oracle: sizes around the tile's edges, corners
at the origin, the world border, around the coordinate beyond which the tables hand over, and far beyond it; both tie rules."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu
CORNERS = [(0, 0), (-8, -8), (8388608 - 4096 - 20, 5), (8388608 - 20, -8388608), (20000000, -17), (-500000000, 530000000),
           (2097100, -2097200), (7499990, -7499990)]
SHAPES = [(1, 1), (32, 32), (33, 63), (31, 2), (130, 97)]


@pytest.mark.parametrize("version", ["26.1", "26.2", "26.3", "26.4-snapshot-2"])
@pytest.mark.parametrize("rule", [0, 2])
def test_nether_tiles(version, rule):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:the_nether", "normal", 0)
    ow = O.World(ge.data_root(), version, "the_nether", "normal")
    rng = np.random.default_rng(8)
    reqs = [(w, int(rng.integers(-2**63, 2**63 - 1)), x - nx // 2, z - nz // 2, nx, nz, int(rng.integers(-5, 40)))
            for x, z in CORNERS for nx, nz in SHAPES]
    plan = mg.Plan(reqs, tie_rule=rule)
    for r, got in zip(reqs, plan.split(plan.run())):
        exp = ow.chunk_grid(*r[1:]) if rule == 2 else ow.quart_grid(*r[1:], O.TIE_ENGINE)
        assert np.array_equal(got, exp), (r[1:], int((got != exp).sum()))
