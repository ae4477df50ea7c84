"""Values that do not fit the tile form's 32-bit fixed point, against the oracle."""
import numpy as np
import pytest

import data_roots
from data_roots import SEED, worlds
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("climate", [{"offset_spline overworld": "S 0 2 -0.5 0.0 C 7.2 0.5 0.0 C 0.1"}, {"offset_spline overworld": "C 7.5"},
                                     {"depth overworld": "-64 320 9.5 -9.5 -0.5"},
                                     {"ridges_folded": "3.5 0.25 -1.0", "offset_spline overworld": "S 3 2 -1.0 0.0 C -0.3 1.0 0.0 C 0.4"}])
def test_values_beyond_the_fixed_point(tmp_path, climate):
    """Offsets, depth gradients and ridges_folded constants whose sums do not fit the tiles' 32-bit values."""
    version = "26.1"
    root = data_roots.make(tmp_path, version, climate)
    mg, w, ow = worlds(root, version, "overworld")
    for qy in (-16, 16, 70):
        q = (-700, 300, 90, 60, qy)
        got, exp = w.quart_grid(*q, mg.TIE_ENGINE), ow.quart_grid(SEED, *q, O.TIE_ENGINE)
        assert np.array_equal(got, exp), int((got != exp).sum())
    got, exp = w.biome_grid(-700, 300, 90, 60, 16, 63), ow.biome_grid(SEED, -700, 300, 90, 60, 16, 63)
    assert np.array_equal(got, exp)
    seeds, pts = np.arange(50), np.random.default_rng(2).integers(-90, 90, (9, 3)).astype(np.int32)
    _, tg = w.seed_points(seeds, pts, want_targets=True)
    _, et = ow.points(seeds, pts, want_targets=True)
    assert np.array_equal(np.asarray(tg).reshape(-1), np.asarray(et).reshape(-1))
