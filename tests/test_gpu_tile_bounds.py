"""The double branch's tile form takes a target only where its error bound settles it, so its exactness rests on those bounds: the
fixed-point noises and the offset spline against the double evaluation, within 2^17 quarts of the origin, beyond, and up to the last
coordinate that the form takes."""
import numpy as np
import pytest

import __graft_entry__ as ge
import data_roots
from data_roots import SEED, worlds
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,dim,preset", [(v, "overworld", p) for v in ("26.1", "26.2") for p in ("normal", "large_biomes", "amplified")] +
                         [("26.1", "the_nether", "normal"), ("26.2", "the_nether", "normal")])
def test_bounds_hold(version, dim, preset):
    mg = ge.package()
    mg.load()
    if mg.device_count() < 1:
        pytest.fail("no CUDA device")
    n = 1 << 22
    for seed in (12345, -(2**62) + 17, 987654321012345):
        w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, preset, seed)
        bad, left, spline_left, worst = mg.check_tile(w, n, seed & 0xFFFF)
        print(f"{version} {dim} {preset} seed {seed}: error / bound {worst[0]:.4f} near, {worst[1]:.4f} far, spline {worst[2]:.4f}; "
              f"open {left / n:.2e}, spline cases open {spline_left / n:.2e}")
        assert bad == 0
        assert max(worst) < 1.0
        assert 0 < left < n // 10  # open cells are evaluated exactly: some, and few


def test_refused():
    mg = ge.package()
    mg.load()
    for version, dim in (("26.3", "overworld"), ("26.1", "the_end")):
        w = mg.Generator.open(ge.data_root(), version).world("minecraft:" + dim, "normal", 1)
        with pytest.raises(mg.McError) as e:
            mg.check_tile(w, 1)
        assert e.value.code == mg.MCGEN_E_ARG


STEEP = ("S 0 5 -1.1 0.0 C 0.044 -0.2 0.0 C 0.3 -0.1999 0.0 S 1 3 -0.5 0.0 C -0.2 0.1 0.0 C 0.25 0.1001 0.0 C -0.1 "
         "0.1 0.0 C 0.02 0.8 0.5 C 0.2")


@pytest.mark.parametrize("version", ["26.1", "26.2"])
def test_steep_spline(tmp_path, version):
    """An offset spline with segments of 1e-4 between far values: its curvature at their ends, 1e8 and more, is what the bound of a
    value near a point has to cover."""
    root = data_roots.make(tmp_path, version, {"offset_spline overworld": STEEP})
    mg, w, ow = worlds(root, version, "overworld")
    bad, left, spline_left, worst = mg.check_tile(w, 1 << 22, 9)
    assert bad == 0 and max(worst) < 1.0, (bad, worst)
    q = (-700, 300, 200, 150, 16)
    assert np.array_equal(w.quart_grid(*q, mg.TIE_ENGINE), ow.quart_grid(SEED, *q, O.TIE_ENGINE))
