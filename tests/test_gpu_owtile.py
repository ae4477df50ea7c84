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


GRIDS = [("26.3", "normal"), ("26.3", "amplified"), ("26.1", "amplified"), ("26.2", "normal")]


def world_pair(version, preset, seed):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    return mg, mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, seed), \
        O.World(ge.data_root(), version, "overworld", preset)


@pytest.mark.parametrize("version,preset", GRIDS)
def test_block_maps_and_points(version, preset):
    """Block maps: the tile form (steps 1 to 4) and the form for sparser samples, at tile edges, at the origin, the world
    border, the coordinate beyond which the tables hand over, and heights inside, at the ends of and outside the build range
    (where the chunk-cell chain is longest); then the same blocks as a list of points."""
    seed = -2757711463728365141
    mg, w, ow = world_pair(version, preset, seed)
    for step in (1, 2, 3, 4, 5, 17):
        for x, z in [(0, 0), (-23, -9), (29999984, -29999984), (4 * 8388608 - 4 * 4096 - 30, 11), (-2000000000, 2000000000)]:
            nx, nz = {1: (67, 35), 2: (33, 18), 3: (1, 40), 4: (50, 7)}.get(step, (17, 16))
            for y in (63, -64, 319, 2000):
                x0, z0 = x - step * nx // 2, z - step * nz // 2
                got, exp = w.biome_grid(x0, z0, nx, nz, step, y), ow.biome_grid(seed, x0, z0, nx, nz, step, y)
                assert np.array_equal(got, exp), (step, x, z, y, int((got != exp).sum()))
        xyz = np.array([(x0 + step * i, y, z0 + step * j) for y in (-80, 40) for j in range(nz) for i in range(nx)], np.int32)
        assert np.array_equal(w.biome_points(xyz), ow.block_points(seed, xyz)), step


@pytest.mark.parametrize("version,preset", GRIDS)
def test_quart_grids_and_chunk_plans(version, preset):
    """Every tie rule's grid form and the chunk-cell plan, one request per world, at the sizes and corners of the batch."""
    seed = 7415553284403671009
    mg, w, ow = world_pair(version, preset, seed)
    shapes = [(1, 1), (17, 33), (250, 40)]
    for x, z in CORNERS:
        for nx, nz in shapes:
            for qy in (16, -17, 90):
                q = (x - nx // 2, z - nz // 2, nx, nz, qy)
                for rule in (mg.TIE_ENGINE, mg.TIE_GRID_CHAIN):
                    assert np.array_equal(w.quart_grid(*q, rule), ow.quart_grid(seed, *q, rule)), (q, rule)
                assert np.array_equal(w.quart_grid(*q, mg.TIE_CHUNK_ORDER), ow.chunk_order_grid(seed, *q)), q
    reqs = [(w, seed, x - nx // 2, z - nz // 2, nx, nz, 15) for x, z in CORNERS for nx, nz in shapes]
    plan = mg.Plan(reqs, tie_rule=mg.TIE_CHUNK_CELL)
    for r, got in zip(reqs, plan.split(plan.run())):
        assert np.array_equal(got, ow.chunk_grid(*r[1:])), r[1:]


@pytest.mark.parametrize("version,dim", [("26.1", "overworld"), ("26.3", "overworld"), ("26.2", "the_nether"), ("26.4-snapshot-2", "the_nether"),
                                         ("26.3", "the_end")])
def test_few_points(version, dim):
    """Point lists around the number whose coordinates travel in the launch, and around the changes of form of the Nether's and the
    Overworld's longer lists."""
    seed = -1
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, "normal", seed)
    ow = O.World(ge.data_root(), version, dim, "normal")
    rng = np.random.default_rng(1)
    for n in (1, 2, 63, 64, 65, 3072, 3073, 8193, 24577):
        xyz = rng.integers(-30000000, 30000000, (n, 3)).astype(np.int32)
        xyz[:, 1] = rng.integers(-100, 400, n)
        assert np.array_equal(w.biome_points(xyz), ow.block_points(seed, xyz)), n
