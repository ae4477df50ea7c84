"""mcgen_gb300_launch_count against the library's own per-kernel profile: the same number of launches for every entry point."""
import numpy as np
import pytest

import __graft_entry__ as ge

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,dim", [("26.1", "overworld"), ("26.3", "overworld"), ("26.1", "the_nether"), ("26.3", "the_end")])
def test_counts_agree(version, dim):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, "normal", 7)
    w.biome_at(0, 64, 0)  # the world's device copies
    rng = np.random.default_rng(1)
    xyz = rng.integers(-3000, 3000, (9000, 3)).astype(np.int32)
    obs = mg.make_obs([(0, 16, 0, list(range(60))), (40, 16, 8, list(range(0, 60, 3)))])
    calls = {"engine": lambda: w.quart_grid(5, 6, 70, 30, 16, mg.TIE_ENGINE),
             "chain": lambda: w.quart_grid(5, 6, 70, 30, 16, mg.TIE_GRID_CHAIN),
             "order": lambda: w.quart_grid(5, 6, 70, 30, 16, mg.TIE_CHUNK_ORDER),
             "map": lambda: w.biome_grid(5, 6, 70, 30, 4, 64), "sparse map": lambda: w.biome_grid(5, 6, 70, 30, 20, 64),
             "point": lambda: w.biome_points(xyz[:1]), "points": lambda: w.biome_points(xyz[:300]),
             "many points": lambda: w.biome_points(xyz), "seeds": lambda: w.seed_points(np.arange(9), xyz[:5]),
             "search": lambda: w.search(obs, kind=mg.SEEDS_RANGE, base=0, n=5000),
             "plan": lambda: mg.Plan([(w, 3, 0, 0, 40, 40, 16)]).run()}
    for name, call in calls.items():
        n0 = mg.launch_count()
        mg.profile(True)
        call()
        mg.profile(False)
        assert mg.launch_count() - n0 == sum(launches for _, launches in mg.profile_read().values()), name
