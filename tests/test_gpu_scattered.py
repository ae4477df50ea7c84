"""Scattered samples searched by whole warps: many seeds at points of any number (last warps partly empty, targets far from
the tree's boxes at extreme heights), and the seed search's observations in both tie modes, against the oracle."""
import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,preset,dim", [("26.1", "normal", "overworld"), ("26.3", "amplified", "overworld"),
                                                ("26.4-snapshot-2", "large_biomes", "overworld"), ("26.2", "normal", "the_nether")])
def test_scattered(version, preset, dim):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, preset, 0)
    ow = O.World(ge.data_root(), version, dim, preset)
    rng = np.random.default_rng(11)
    for ns, npt in ((1, 1), (1, 31), (3, 11), (129, 1), (17, 9)):
        seeds = rng.integers(-2**63, 2**63 - 1, ns)
        pts = rng.integers(-7000, 7000, (npt, 3)).astype(np.int32)
        pts[:, 1] = rng.integers(-600, 600, npt)
        got, tg = w.seed_points(seeds, pts, want_targets=True)
        exp, et = ow.points(seeds, pts, want_targets=True)
        assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(exp).reshape(-1)), (ns, npt)
        assert np.array_equal(np.asarray(tg).reshape(-1), np.asarray(et).reshape(-1)), (ns, npt)
    seeds = rng.integers(-2**63, 2**63 - 1, 777)
    at = rng.integers(-3000, 3000, (3, 3)).astype(np.int32)
    at[:, 1] = (16, -200, 300)
    ids = np.asarray(ow.points(seeds[:1], at)).reshape(-1)
    obs = mg.make_obs([(int(x), int(y), int(z), [int(b)]) for (x, y, z), b in zip(at, ids)])
    oobs = O.make_obs([(int(x), int(y), int(z), [int(b)]) for (x, y, z), b in zip(at, ids)])
    for ties in (False, True):
        got = w.search(obs, kind=mg.SEEDS_LIST, seeds=seeds, ties=ties)
        exp = ow.search(oobs, kind=O.SEEDS_LIST, seeds=seeds, ties=ties)
        assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1]), (ties, got[1], exp[1])


@pytest.mark.parametrize("version,preset", [("26.1", "normal"), ("26.3", "amplified"), ("26.4-snapshot-2", "normal")])
def test_search_stages(version, preset):
    """Enough candidates for several staged observations and the rest by a warp each; masks of one common biome, of many and of
    none (the table of possible biomes all clear), block observations."""
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, 0)
    ow = O.World(ge.data_root(), version, "overworld", preset)
    rng = np.random.default_rng(5)
    n, base = 6001, int(rng.integers(-2**63, 2**63 - 1))
    for block in (False, True):
        scale = 4 if block else 1
        at = rng.integers(-3000, 3000, (4, 3)) * scale
        at[:, 1] = np.array([16, 16, -9, 60]) * scale
        ids = [int(b) for b in np.asarray(ow.points([base + 7], at // scale)).reshape(-1)]
        masks = [sorted(set(ids) | set(range(0, 60, 2))), list(range(60)), [ids[2], ids[0]], [ids[3]]]
        for rows in (masks, [[127]] + masks[1:]):
            r = [(int(x), int(y), int(z), m) for (x, y, z), m in zip(at, rows)]
            got = w.search(mg.make_obs(r, block), kind=mg.SEEDS_RANGE, base=base, n=n)
            exp = ow.search(O.make_obs(r, block), kind=O.SEEDS_RANGE, base=base, n=n)
            assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1]), (block, got[1], exp[1])


@pytest.mark.parametrize("version", ["26.1", "26.3"])
def test_end_tiles(version):
    """End grids of every tile shape: one chunk, sides around a tile's 24 chunks and their equal parts, corners inside a chunk, at the
    central disc, at the world border and beyond the fixed-point skew's range; batched and alone."""
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    seed = 7126353871628162251
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:the_end", "normal", seed)
    ow = O.World(ge.data_root(), version, "the_end", "normal")
    shapes = [(1, 1), (3, 97), (96, 97), (101, 5), (200, 130)]
    corners = [(0, 0), (-257, 250), (1001, -3002), (7499990, -7499990), (4 * (1 << 21) - 60, 77), (-20000003, 30000001)]
    reqs = [(w, seed, x - nx // 2, z - nz // 2, nx, nz, 16) for x, z in corners for nx, nz in shapes]
    plan = mg.Plan(reqs)
    for r, got in zip(reqs, plan.split(plan.run())):
        exp = ow.quart_grid(*r[1:], O.TIE_ENGINE)
        assert np.array_equal(got, exp), r[1:]
        assert np.array_equal(w.quart_grid(*r[2:]), exp), r[1:]


def test_nether_rejected_draws():
    """About one seed in 12,000 rejects a draw in a shuffle of its Nether noises, which moves the octaves built after it."""
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), "26.3").world("minecraft:the_nether", "normal", 0)
    ow = O.World(ge.data_root(), "26.3", "the_nether", "normal")
    seeds = np.random.default_rng(2).integers(-2**63, 2**63 - 1, 120000)
    pts = np.array([[137, 16, -911]], np.int32)
    _, tg = w.seed_points(seeds, pts, want_targets=True)
    _, et = ow.points(seeds, pts, want_targets=True)
    assert np.array_equal(np.asarray(tg).reshape(-1, 6), np.asarray(et).reshape(-1, 6))


@pytest.mark.parametrize("version,preset", [("26.1", "normal"), ("26.2", "amplified"), ("26.1", "large_biomes")])
def test_seed_targets_fixed_point(version, preset):
    """The double branch's targets from fixed point: points around the flush of kept values, beyond the tables' coordinates (the
    exact form), near and beyond 2^17, extreme heights; seeds around a block's number."""
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, 0)
    ow = O.World(ge.data_root(), version, "overworld", preset)
    rng = np.random.default_rng(4)
    lims = (300, 131060, 131090, 7499990, 8388607, 500000000)
    for ns, npt in ((5, 129), (1, 64), (3, 65), (41, 9), (4, 8)):
        seeds = rng.integers(-2**63, 2**63 - 1, ns)
        lim = np.array([lims[i % 6] for i in range(npt)])
        pts = np.stack([rng.integers(-lim, lim), rng.integers(-90, 90, npt), rng.integers(-lim, lim)], 1).astype(np.int32)
        if npt == 129: pts[:64, [0, 2]] = 8388600  # a full queue
        got, tg = w.seed_points(seeds, pts, want_targets=True)
        exp, et = ow.points(seeds, pts, want_targets=True)
        assert np.array_equal(np.asarray(tg).reshape(-1, 6), np.asarray(et).reshape(-1, 6)), (ns, npt)
        assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(exp).reshape(-1)), (ns, npt)
        assert np.array_equal(np.asarray(w.seed_points(seeds, pts)).reshape(-1), np.asarray(exp).reshape(-1)), (ns, npt)
