"""Box queries and refits at the edges of their kernels: query sets around a warp over trees of a few leaves
(every part of a split walk, leaves above the split's depth), the same EF pairs whatever the order of the
edge queries, and a tree whose top nodes pass the shared-memory forms' bounds. Pair sets,
topology and boxes equal the oracle's."""
import types

import numpy as np
import pytest
import torch

from test_lbvh_gpu import _assert_tree_equal, _build_both, _dev, _sorted_pairs
from untangling26_b200 import synthetic
from untangling26_b200.intersection_resolver import CollisionScene
from untangling26_b200.lbvh import TREE_FACE, TREE_VERT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [2, 3, 5, 33, 1025])
@pytest.mark.parametrize("queries", [1, 31, 32, 33, 200])
@pytest.mark.parametrize("mode", [0, 2])
def test_small_query_sets(oracle, u26ctx, leaves, queries, mode):
    rng = np.random.default_rng(1000 * leaves + queries)
    nv = max(3 * leaves, 2 * queries)
    x = rng.uniform(-1, 1, (nv, 3)).astype(np.float32)
    faces = np.arange(3 * leaves, dtype=np.uint32).reshape(-1, 3)
    edges = rng.permutation(nv)[:2 * queries].astype(np.uint32).reshape(-1, 2)
    xq = x if mode == 2 else x[:queries].copy()
    m = types.SimpleNamespace(x=x, faces=faces, edges=edges, num_verts=nv, num_faces=leaves, num_edges=queries)
    ot, t, (dx, _, dth, _) = _build_both(oracle, u26ctx, TREE_FACE, m)
    d_hat = np.full(nv, 1e-3, np.float32)
    th = np.zeros(nv, np.float32)
    ref, total, _ = oracle.lbvh_query(ot, mode, xq, xq, edges, d_hat, th)
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((total + 8, 2), dtype=torch.int32, device="cuda")
    dq = _dev(xq)
    if mode == 0:
        t.broad_phase_query_from_verts(dq, dq, count, pairs, _dev(d_hat), dth)
    else:
        t.broad_phase_query_from_edges_unculled(dq, dq, _dev(edges), count, pairs, _dev(d_hat), dth)
    assert int(count.item()) == total
    assert np.array_equal(_sorted_pairs(pairs[:total].cpu().numpy().view(np.uint32)), _sorted_pairs(ref))
    assert u26ctx.device_errors() == 0


@pytest.mark.parametrize("n", [5, 24, 90])
def test_ef_pairs_of_any_edge_order(oracle, u26ctx, n):
    m = synthetic.folded_sheet(n, seed=3)
    ef, idx = oracle.detect_ef(m)
    sc = CollisionScene(u26ctx, m)
    sc.construct_lbvh()
    for order in (sc.edge_order, None, torch.randperm(m.num_edges, device="cuda").int()):
        sc.edge_order = order
        sc.detect_ef_fused()
        got, got_idx = sc.ef_pairs()
        assert np.array_equal(got_idx, idx) and got.tobytes() == ef.tobytes()
    assert u26ctx.device_errors() == 0


def test_refit_of_many_top_nodes(oracle, u26ctx):
    """9 M leaves: about 13,500 nodes of more than 1,024 leaves, past the 7,168 and 12,288 that the one-block
    kernels keep in shared memory."""
    n = 9_000_000
    rng = np.random.default_rng(9)
    x = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    m = types.SimpleNamespace(x=x, faces=None, edges=None, num_verts=n, num_faces=0, num_edges=0)
    ot, t, _ = _build_both(oracle, u26ctx, TREE_VERT, m)
    assert t.check_health()
    _assert_tree_equal(ot, t.arrays())
