"""The batched form's Overworld tile kernels (16 x 16-cell tiles reading tables of lattice nodes) against the oracle:
sizes around the tile's edges, corners at the origin (sums in (-1, 0), fractions near 0), at the world border, around the
coordinate beyond which the tables hand the tile to the per-cell form, and far beyond it."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu
CORNERS = [(0, 0), (-8, -8), (8388608 - 4096 - 20, 5), (8388608 - 20, -8388608), (20000000, -17), (-500000000, 530000000),
           (2097100, -2097200), (7499990, -7499990)]
SHAPES = [(1, 1), (16, 16), (17, 33), (40, 5), (15, 1), (250, 130)]


@pytest.mark.parametrize("version,preset", [("26.3", "normal"), ("26.3", "amplified"), ("26.4-snapshot-2", "large_biomes"),
                                            ("26.1", "normal"), ("26.2", "large_biomes"), ("26.1", "amplified")])
def test_overworld_tiles(version, preset):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, 0)
    ow = O.World(ge.data_root(), version, "overworld", preset)
    rng = np.random.default_rng(3)
    reqs = [(w, int(rng.integers(-2**63, 2**63 - 1)), x - nx // 2, z - nz // 2, nx, nz, int(rng.integers(-20, 85)))
            for x, z in CORNERS for nx, nz in SHAPES]
    plan = mg.Plan(reqs)
    for r, got in zip(reqs, plan.split(plan.run())):
        exp = ow.quart_grid(*r[1:], O.TIE_ENGINE)
        assert np.array_equal(got, exp), (r[1:], int((got != exp).sum()))
