"""The warp-shared tree search over a table whose last group of clustered leaves is partly empty, against the 64-bit search and the
oracle."""
import numpy as np
import pytest

import data_roots
from data_roots import SEED, worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version", ["26.1", "26.3", "26.4-snapshot-2"])
def test_no_leaf_near_the_origin(tmp_path, version):
    """Every leaf 20,000 away in the last dimension (the nearest ones stay the same), the last group of clustered leaves partly
    empty: what lies in its empty places must not bound a search."""
    def far(rows):
        rows = rows[:1001]
        for r in rows:
            r[12] = 20000
        return rows

    root = data_roots.make(tmp_path, version, params={"overworld": far})
    mg, w, ow = worlds(root, version, "overworld")
    assert mg.check_tree(w, 1 << 20, 5) == (0, 0)
    for step in (4, 16):
        got, exp = w.biome_grid(-3000, 500, 200, 100, step, 0), ow.biome_grid(SEED, -3000, 500, 200, 100, step, 0)
        assert np.array_equal(got, exp), (step, int((got != exp).sum()))
