"""Tables of one entry."""
import pytest

import data_roots
from data_roots import compare_all, worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,dim", [("26.1", "overworld"), ("26.3", "overworld"), ("26.3", "the_nether")])
def test_one_leaf(tmp_path, version, dim):
    """A table of one entry: its biome everywhere."""
    root = data_roots.make(tmp_path, version, params={"overworld" if dim == "overworld" else "nether": lambda rows: rows[:1]})
    compare_all(*worlds(root, version, dim))
