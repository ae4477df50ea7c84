"""Cells that the tiles leave open are recorded for a later launch; those beyond the record, or all of them where there is none, are
evaluated in place.  Areas beyond the coordinates of the double branch's tables: left open where they are few, by a thread each in
the tile where they are many."""
import numpy as np
import pytest

import __graft_entry__ as ge
import data_roots
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SEED = -6543217890123


def pair(version, preset="normal"):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    return mg, mg.Generator.open(ge.data_root(), version).world("minecraft:overworld", preset, SEED), \
        O.World(ge.data_root(), version, "overworld", preset)


@pytest.mark.parametrize("version,preset", [("26.1", "normal"), ("26.2", "amplified")])
@pytest.mark.parametrize("step", [1, 4, 5, 17])
def test_maps_beyond_the_coordinates(version, preset, step):
    mg, w, ow = pair(version, preset)
    nx, nz = 117, 81
    x0, z0 = 4 * 8388608 + 30, -17
    got, exp = w.biome_grid(x0, z0, nx, nz, step, 40), ow.biome_grid(SEED, x0, z0, nx, nz, step, 40)
    assert np.array_equal(got, exp), int((got != exp).sum())


@pytest.mark.parametrize("version", ["26.1", "26.2"])
def test_grids_beyond_the_coordinates(version):
    mg, w, ow = pair(version)
    x0 = 8388608 - 4096
    for q in ((x0, -5, 60, 68, 16), (x0, -5, 61, 68, 16), (x0 - 40, -5, 120, 75, 16), (-x0 - 200, 9, 200, 90, -3), (7, x0 - 1, 70, 60, 20)):
        for rule in (mg.TIE_ENGINE, mg.TIE_GRID_CHAIN):
            assert np.array_equal(w.quart_grid(*q, rule), ow.quart_grid(SEED, *q, rule)), (q, rule)
        assert np.array_equal(w.quart_grid(*q, mg.TIE_CHUNK_ORDER), ow.chunk_order_grid(SEED, *q)), q
        for tie in (mg.TIE_ENGINE, mg.TIE_CHUNK_CELL):
            got = mg.Plan([(w, SEED, *q)], tie_rule=tie).run().reshape(q[3], q[2])
            exp = ow.chunk_grid(SEED, *q) if tie == mg.TIE_CHUNK_CELL else ow.quart_grid(SEED, *q, O.TIE_ENGINE)
            assert np.array_equal(got, exp), (q, tie)


def test_grids_beyond_the_record(tmp_path):
    """An offset spline so steep everywhere that most targets stay open."""
    points = " ".join(f"{-1.2 + 0.01 * i:.2f} 0.0 C {3 - 6 * (i % 2)}.0" for i in range(241))
    root = data_roots.make(tmp_path, "26.1", {"offset_spline overworld": "S 0 241 " + points})
    mg, w, ow = data_roots.worlds(root, "26.1", "overworld", SEED)
    q = (-300, 55, 131, 97, 16)  # 12,707 cells, room for 4,493
    for rule in (mg.TIE_ENGINE, mg.TIE_GRID_CHAIN):
        assert np.array_equal(w.quart_grid(*q, rule), ow.quart_grid(SEED, *q, rule)), rule
    for tie in (mg.TIE_ENGINE, mg.TIE_CHUNK_CELL):
        got = mg.Plan([(w, SEED, *q)], tie_rule=tie).run().reshape(q[3], q[2])
        assert np.array_equal(got, ow.chunk_grid(SEED, *q) if tie == mg.TIE_CHUNK_CELL else ow.quart_grid(SEED, *q, O.TIE_ENGINE)), tie
    for step in (4, 17):
        assert np.array_equal(w.biome_grid(0, 0, 131, 97, step, 63), ow.biome_grid(SEED, 0, 0, 131, 97, step, 63)), step
    seeds, pts = np.arange(9), np.random.default_rng(2).integers(-90, 90, (70, 3)).astype(np.int32)
    _, tg = w.seed_points(seeds, pts, want_targets=True)
    _, et = ow.points(seeds, pts, want_targets=True)
    assert np.array_equal(np.asarray(tg).reshape(-1), np.asarray(et).reshape(-1))


@pytest.mark.parametrize("version", ["26.1", "26.3"])
def test_server_without_room_for_the_record(version):
    """A batch whose record cannot be allocated (injected on the host) is served all the same."""
    mg, w, ow = pair(version)
    srv = mg.Server(hbm_budget_bytes=64 << 20, max_inflight=1)
    try:
        for q in ((8388600, 4, 90, 70, 16), (-300, 77, 90, 70, 16), (8388600, 4, 33, 20, 16)):
            srv.fail_next(mg.FAIL_RECORD)
            ids, _ = srv.wait(srv.submit(w, SEED, *q))
            assert np.array_equal(ids, ow.quart_grid(SEED, *q, O.TIE_ENGINE)), q
        ids, _ = srv.wait(srv.submit(w, SEED, -300, 77, 90, 70, 16))  # and with the record again
        assert np.array_equal(ids, ow.quart_grid(SEED, -300, 77, 90, 70, 16, O.TIE_ENGINE))
    finally:
        srv.close()
