"""Many seeds x points of the double branch: samples that the fixed point leaves open are queued per seed and evaluated at the end of
each run of 64 points.  Queues of very different lengths (none, one, all 64) in the seeds of one block, emptied several times, in
many blocks at once, again and again: the same targets each time, the oracle's."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,preset", [("26.1", "normal"), ("26.2", "amplified")])
def test_queues_emptied_many_times(version, preset):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, 0)
    ow = O.World(ge.data_root(), version, "overworld", preset)
    rng = np.random.default_rng(6)
    npt = 4 * 64 + 3
    pts = rng.integers(-2500, 2500, (npt, 3)).astype(np.int32)
    pts[:, 1] = rng.integers(-16, 81, npt)
    pts[64:128, 0] = 8388606  # beyond the tables' coordinates: all 64 are queued
    pts[200, 2] = -8388606
    seeds = rng.integers(-2**63, 2**63 - 1, 2003)
    first = None
    for _ in range(4):
        _, tg = w.seed_points(seeds, pts, want_targets=True)
        tg = np.asarray(tg).reshape(len(seeds), npt, 6)
        if first is None:
            first = tg
            _, et = ow.points(seeds[-150:], pts, want_targets=True)
            assert np.array_equal(tg[-150:], np.asarray(et).reshape(150, npt, 6))
        else:
            assert np.array_equal(tg, first)
