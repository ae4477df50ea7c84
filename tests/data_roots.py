"""Data roots of the tests' own: copies of the shipped data with some lines replaced."""
import os
import shutil

import numpy as np
import pytest

import __graft_entry__ as ge
from oracle import oracle as O

SEED = 4215570217845711903


def make(tmp_path, version, climate=None, params=None):
    """A copy of `version`'s data under tmp_path.  climate: {line prefix: new line} of the climate file; params: {dimension file's
    name: function of its list of rows (lists of strings)}."""
    src, dst = os.path.join(ge.data_root(), "data"), tmp_path / "data"
    shutil.copytree(os.path.join(src, "params", version), dst / "params" / version)
    with open(os.path.join(src, f"climate-{version}.txt")) as f:
        lines = f.read().splitlines()
    for prefix, line in (climate or {}).items():
        at = [i for i, ln in enumerate(lines) if ln.startswith(prefix + " ")]
        assert len(at) == 1, prefix
        lines[at[0]] = f"{prefix} {line}"
    (dst / f"climate-{version}.txt").write_text("\n".join(lines) + "\n")
    for name, change in (params or {}).items():
        f = dst / "params" / version / f"{name}.tsv"
        rows = [ln.split("\t") for ln in f.read_text().splitlines() if ln and ln[0] != "#"]
        f.write_text("\n".join("\t".join(map(str, r)) for r in change(rows)) + "\n")
    return str(tmp_path)


def noise(version, first, amplitudes):
    """The fields after a noise's name."""
    amps = " ".join(f"{a:.1f}" for a in amplitudes)
    return f"0 {first} {len(amplitudes)} 0 0 0 {amps}" if version < "26.3" else f"1 {first} {len(amplitudes)} 0.95 1 1 {amps}"


def worlds(root, version, dim, seed=SEED):
    """The binding, and the world of a data root in the library and in the oracle."""
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    return mg, mg.Generator.open(root, version).world("minecraft:" + dim, "normal", seed), O.World(root, version, dim, "normal")


def compare_all(mg, w, ow, y=63, search=True):
    """Every entry point on small areas: at the origin and off it, odd sizes.  search: whether it may be asked."""
    rng = np.random.default_rng(21)
    for x, z, nx, nz in ((-19, 7, 37, 18), (4000, -3001, 5, 70)):
        q = (x, z, nx, nz, 16)
        for rule in (mg.TIE_ENGINE, mg.TIE_GRID_CHAIN):
            assert np.array_equal(w.quart_grid(*q, rule), ow.quart_grid(SEED, *q, rule)), (q, rule)
        assert np.array_equal(w.quart_grid(*q, mg.TIE_CHUNK_ORDER), ow.chunk_order_grid(SEED, *q)), q
        for step in (1, 4, 16, 37):
            got, exp = w.biome_grid(x, z, nx, nz, step, y), ow.biome_grid(SEED, x, z, nx, nz, step, y)
            assert np.array_equal(got, exp), (x, z, step, int((got != exp).sum()))
    reqs = [(w, int(rng.integers(-2**63, 2**63 - 1)), x, z, nx, nz, 16) for x, z, nx, nz in
            ((0, 0, 1, 1), (-8, -8, 33, 17), (9000, -9000, 40, 70))]
    for rule in (mg.TIE_ENGINE, mg.TIE_CHUNK_CELL):
        plan = mg.Plan(reqs, tie_rule=rule)
        for shape in range(4):
            plan.shape = shape
            for r, got in zip(reqs, plan.split(plan.run())):
                exp = ow.chunk_grid(*r[1:]) if rule == mg.TIE_CHUNK_CELL else ow.quart_grid(*r[1:], O.TIE_ENGINE)
                assert np.array_equal(got, exp), (rule, shape, r[1:])
    for n in (1, 64, 300, 8200):
        xyz = rng.integers(-30000, 30000, (n, 3)).astype(np.int32)
        xyz[:, 1] = y
        assert np.array_equal(w.biome_points(xyz), ow.block_points(SEED, xyz)), n
    seeds, pts = rng.integers(-2**63, 2**63 - 1, 37), rng.integers(-3000, 3000, (11, 3)).astype(np.int32)
    pts[:, 1] = 16
    got, tg = w.seed_points(seeds, pts, want_targets=True)
    exp, et = ow.points(seeds, pts, want_targets=True)
    assert np.array_equal(np.asarray(tg).reshape(-1), np.asarray(et).reshape(-1))
    assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(exp).reshape(-1))
    if not search:
        return
    ids = np.asarray(ow.points([SEED], pts[:3])).reshape(-1)
    rows = [(int(x), 16, int(z), [int(b)]) for (x, _, z), b in zip(pts[:3], ids)]
    for ties in (False, True):
        got = w.search(mg.make_obs(rows), kind=mg.SEEDS_RANGE, base=SEED - 700, n=1500, ties=ties)
        exp = ow.search(O.make_obs(rows), kind=O.SEEDS_RANGE, base=SEED - 700, n=1500, ties=ties)
        assert np.array_equal(got[0], exp[0]) and np.array_equal(got[1], exp[1]), (ties, got[1], exp[1])
        assert SEED in got[0]
