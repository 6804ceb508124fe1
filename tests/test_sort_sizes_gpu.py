"""The device sort through LBVH construction at its edges: the one-block form up to 8,192 keys, tiles of
3,072 keys above it, and points that share Morton codes (the order of equal codes is the
leaf order). Keys, order and topology equal the oracle's."""
import types

import numpy as np
import pytest

from test_lbvh_gpu import _assert_tree_equal, _build_both
from untangling26_b200.lbvh import TREE_VERT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 127, 128, 129, 1023, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 9215, 9216, 9217, 12289, 250_001])
@pytest.mark.parametrize("spread", ["uniform", "few codes"])
def test_sorted_order(oracle, u26ctx, n, spread):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1.0, 1.0, (n, 3))
    if spread == "few codes":
        x = rng.integers(0, 5, (n, 3)) * 0.25 + 0.01 * (np.arange(n) % 3 == 0)[:, None]
    m = types.SimpleNamespace(x=x.astype(np.float32), faces=None, edges=None, num_verts=n, num_faces=0, num_edges=0)
    ot, t, _ = _build_both(oracle, u26ctx, TREE_VERT, m)
    _assert_tree_equal(ot, t.arrays())
    assert t.check_health()
