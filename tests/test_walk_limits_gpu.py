"""Box queries that meet the 32-entry stack or the 100,000 step bound, as small query sets (which are walked in
parts of the tree where neither can be met): the pairs that a stopped query has found by then and the error flags are the
oracle's. The deep tree is a chain of Morton prefixes 01..1, then of id prefixes 1..1, with two leaves beside
every link, so its stack fills with siblings; a cluster at the code's other half is walked first."""
import types

import numpy as np
import pytest
import torch

from test_lbvh_gpu import _build_both, _dev, _sorted_pairs
from untangling26_b200 import Context
from untangling26_b200._native import DEVERR_ITERATION_CAP, DEVERR_STACK_OVERFLOW
from untangling26_b200.intersection_resolver import CollisionScene
from untangling26_b200.lbvh import TREE_FACE, TREE_VERT
from untangling26_b200.mesh import Mesh

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    c = Context(0)
    yield c
    c.close()


def _codes(n, links):
    """A Morton code for each of n leaves (n a power of two): `links` links of the chain."""
    bits = int(np.log2(n))
    code = np.zeros(n, np.int64)
    ones = (1 << 29) - 1
    at_end = np.zeros(n, bool)
    for k in range(bits - 1):
        first = ((1 << k) - 1) << (bits - k)  # ids 1..1 0..0
        at_end[first:first + 2] = True
    at_end[n - 2:] = True
    free = np.flatnonzero(~at_end)
    code[at_end] = ones if links > 29 else ones >> (29 - links) << (29 - links)
    code[free] = (1 << 29) + np.arange(len(free)) // 2 * ((1 << 29) // len(free))  # the other half, two by two
    for b in range(min(links, 29)):
        code[free[2 * b:2 * b + 2]] = (ones >> (29 - b)) << (29 - b)  # 0 1..1 0..0
    return code


def _centres(code):
    cell = np.zeros((len(code), 3), np.int64)
    for i in range(10):
        for a in range(3):
            cell[:, a] |= ((code >> (3 * i + 2 - a)) & 1) << i
    return (cell + 0.5) / 1024.0


def _soup(links, n, size):
    """Small triangles at the chain's centres, and one at each corner of the box."""
    rng = np.random.default_rng(links)
    c = _centres(_codes(n, links))
    x = (c[:, None] + rng.uniform(-size, size, (n, 3, 3))).reshape(-1, 3)
    x = np.concatenate([x, np.repeat([[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]], 3, 0)]).astype(np.float32)
    return x, np.arange(3 * n + 6, dtype=np.uint32).reshape(-1, 3)


def _height(ot):
    ni = ot.n - 1
    front, h = np.array([0]), 0
    while len(front):
        front = ot.children[front].reshape(-1)
        front = front[front < ni]
        h += 1
    return h


@pytest.mark.parametrize("n", [1024, 8192])
@pytest.mark.parametrize("links", [12, 20, 23, 24, 29, 30])
@pytest.mark.parametrize("mode", [0, 2])
def test_stack_of_deep_trees(oracle, ctx, n, links, mode):
    x, faces = _soup(links, n, 1.5e-4)
    edges = np.stack([faces[:, 0], faces[:, 1]], 1)[:200].copy()
    m = types.SimpleNamespace(x=x, faces=faces, edges=edges, num_verts=len(x), num_faces=len(faces), num_edges=len(edges))
    ot, t, (_, _, dth, _) = _build_both(oracle, ctx, TREE_FACE, m)
    assert t.check_health()
    # every third query covers the tree, the others have boxes of their own size
    d_hat = np.where(np.arange(m.num_verts) // 3 % 3 == 0, 4.0, 0.01).astype(np.float32)
    xq = m.x if mode == 2 else m.x[:300].copy()
    ref, total, overflow = oracle.lbvh_query(ot, mode, xq, xq, m.edges, d_hat, np.zeros(m.num_verts, np.float32))
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((total + 8, 2), dtype=torch.int32, device="cuda")
    dq = _dev(xq)
    if mode == 0:
        t.broad_phase_query_from_verts(dq, dq, count, pairs, _dev(d_hat), dth)
    else:
        t.broad_phase_query_from_edges_unculled(dq, dq, _dev(m.edges), count, pairs, _dev(d_hat), dth)
    assert int(count.item()) == total
    assert np.array_equal(_sorted_pairs(pairs[:total].cpu().numpy().view(np.uint32)), _sorted_pairs(ref))
    assert (ctx.device_errors() == DEVERR_STACK_OVERFLOW) if overflow else (ctx.device_errors() == 0)
    if links == 12:
        assert not overflow and _height(ot) <= 32
    if links == 30:
        assert overflow and _height(ot) > 32 and total > 0


@pytest.mark.parametrize("links", [12, 30])
def test_fused_detection_of_deep_trees(oracle, ctx, links):
    m = Mesh(*_soup(links, 1024, 4e-4))
    sc = CollisionScene(ctx, m, d_hat=2.0, parity_tree=True)
    sc.construct_lbvh()
    sc.detect_ef_fused()
    got, got_idx = sc.ef_pairs()
    flags = ctx.device_errors()
    ot = oracle.lbvh_build(TREE_FACE, m.x, m.faces, num_verts=m.num_verts)
    th, d_hat = np.zeros(m.num_verts, np.float32), np.full(m.num_verts, 2.0, np.float32)
    oracle.lbvh_refit(ot, m.x, m.x, th, m.faces)
    broad, _, overflow = oracle.lbvh_query(ot, 2, m.x, m.x, m.edges, d_hat, th)
    ef, idx = oracle.ef_narrow(broad, m.x, m.edges, m.faces, d_hat)
    assert len(idx) > 0
    assert bool(overflow) == (links == 30)
    assert flags == (DEVERR_STACK_OVERFLOW if overflow else 0)
    assert np.array_equal(got_idx, idx) and got.tobytes() == ef.tobytes()
    sc.close()


@pytest.mark.parametrize("n", [100001, 100002, 120000])
def test_steps_of_queries_over_many_leaves(oracle, ctx, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    m = types.SimpleNamespace(x=x, faces=None, edges=None, num_verts=n, num_faces=0, num_edges=0)
    ot, t, (_, _, dth, _) = _build_both(oracle, ctx, TREE_VERT, m)
    xq = x[:7].copy()
    d_hat = np.array([5.0, 0.1, 5.0, 0.01, 5.0, 0.5, 0.3] + [0.0] * (n - 7), np.float32)
    ref, total, overflow = oracle.lbvh_query(ot, 0, xq, xq, None, d_hat, np.zeros(n, np.float32))
    assert overflow == 0
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((total + 8, 2), dtype=torch.int32, device="cuda")
    dq = _dev(xq)
    t.broad_phase_query_from_verts(dq, dq, count, pairs, _dev(d_hat), dth)
    assert int(count.item()) == total
    assert np.array_equal(_sorted_pairs(pairs[:total].cpu().numpy().view(np.uint32)), _sorted_pairs(ref))
    assert ctx.device_errors() == (DEVERR_ITERATION_CAP if n > 100001 else 0)
