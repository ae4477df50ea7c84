"""Worlds from data that no shipped version has, against the oracle: those that the tile forms do not take, so that the general forms
of grids, batches, seed points and the search run (they do for no shipped world), and tables of ties."""
import numpy as np
import pytest

import data_roots
from data_roots import SEED, compare_all, worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version", ["26.1", "26.3"])
def test_four_shift_octaves(tmp_path, version):
    """More shift octaves than the Overworld tiles hold: the per-cell forms of everything."""
    root = data_roots.make(tmp_path, version, {"noise offset": data_roots.noise(version, -3, (1, 1, 1, 1))})
    compare_all(*worlds(root, version, "overworld"))


@pytest.mark.parametrize("version", ["26.2", "26.3"])
def test_nine_shift_octaves(tmp_path, version):
    """More shift octaves than a warp has lanes for both shift noises (and than the fused seed kernels take)."""
    root = data_roots.make(tmp_path, version, {"noise offset": data_roots.noise(version, -9, (1,) * 9),
                                               "noise continentalness": data_roots.noise(version, -9, (1, 1, 2, 2))})
    mg, w, ow = worlds(root, version, "overworld")
    compare_all(mg, w, ow, search=False)
    with pytest.raises(mg.McError) as e:
        w.search(mg.make_obs([(0, 16, 0, [1])]), kind=mg.SEEDS_RANGE, base=0, n=10)
    assert e.value.code == mg.MCGEN_E_UNSUPPORTED


@pytest.mark.parametrize("version", ["26.1", "26.3"])
@pytest.mark.parametrize("amplitudes", [(1, 1, 1, 1), (1, 0, 0, 1, 1), (0, 1)])
def test_other_nether_octaves(tmp_path, version, amplitudes):
    """Nether noises of more and other octaves than the game's: the per-cell form, lattices built by one lane (eight and six
    octaves of a noise with the first one; absent ones are skipped)."""
    root = data_roots.make(tmp_path, version, {"noise nether/temperature": data_roots.noise(version, -len(amplitudes) + 1, amplitudes)})
    compare_all(*worlds(root, version, "the_nether"))


@pytest.mark.parametrize("version,dim", [("26.1", "overworld"), ("26.3", "overworld"), ("26.2", "the_nether"), ("26.3", "the_nether")])
def test_every_cell_tied(tmp_path, version, dim):
    """Each leaf twice, with two biomes: every cell is tied, so the tiles leave all of them open and the record of open cells is
    full long before the last tile."""
    def twice(rows):
        rows = rows[::7] if dim == "overworld" else rows
        return rows + [r[:13] + ["minecraft:plains"] for r in rows]

    root = data_roots.make(tmp_path, version, params={"overworld" if dim == "overworld" else "nether": twice})
    mg, w, ow = worlds(root, version, dim)
    y0 = -64 if dim == "overworld" else 0  # the column's lowest cells: short chains
    compare_all(mg, w, ow, y=y0, search=False)
    for step in (4, 16):
        got, exp = w.biome_grid(-200, -333, 131, 97, step, y0), ow.biome_grid(SEED, -200, -333, 131, 97, step, y0)
        assert np.array_equal(got, exp), (step, int((got != exp).sum()))
    reqs = [(w, SEED, -65, 40, 131, 97, y0 >> 2)]
    plan = mg.Plan(reqs, tie_rule=mg.TIE_CHUNK_CELL)
    assert np.array_equal(plan.split(plan.run())[0], ow.chunk_grid(*reqs[0][1:]))
