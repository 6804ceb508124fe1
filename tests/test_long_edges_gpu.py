"""Ray casting of meshes whose edges are hundreds to thousands of units long (a sheet modelled in millimetres): the
batched form's node tests keep every edge that the plain form's per-request walk tests, so both forms return
the same supports and results. Sheet A's long edges end exactly where edges of sheet B cross them, near the
origin, where a node's margin is small beside the rounding of the swept edge's far bound."""
import numpy as np
import pytest

from untangling26_b200.intersection_resolver import CollisionScene
from untangling26_b200.mesh import Mesh
from untangling26_b200.prp import prp_params

pytestmark = pytest.mark.gpu


def _mesh(length, seed, axis, rows=17, cols=12):
    """Sheet A at z = 0: every row is one edge from -length to a seeded end in [0.3, 0.5], then short edges. Sheet B has
    two rows around each of A's, at the same x, and a dent through A."""
    rng = np.random.default_rng(seed)
    ends = rng.uniform(0.3, 0.5, rows)
    y, s = np.linspace(0.0, 1.0, rows), 0.3 / (rows - 1)
    step = np.linspace(0.0, 0.5, cols)

    def sheet(ys, es, height):
        px = np.concatenate([np.full((len(ys), 1), -float(length)), es[:, None] + step[None]], 1)
        py = np.broadcast_to(ys[:, None], px.shape)
        i, c = np.meshgrid(np.arange(len(ys) - 1), np.arange(cols), indexing="ij")
        a = (i * (cols + 1) + c).reshape(-1)
        b = a + cols + 1
        faces = np.stack([a, b, b + 1, a, b + 1, a + 1], 1).reshape(-1, 3)
        return np.stack([px, py, height(px, py)], 2).reshape(-1, 3), faces

    xa, fa = sheet(y, ends, lambda u, v: 0.0 * u)
    xb, fb = sheet(np.stack([y - s, y + s], 1).reshape(-1), np.repeat(ends, 2),
                   lambda u, v: 0.02 - 0.1 * np.exp(-((u - 0.55) ** 2 + (v - 0.5) ** 2) / 0.02))
    x = np.roll(np.concatenate([xa, xb]), axis, axis=1).astype(np.float32)
    faces = np.concatenate([fa, fb + len(xa)]).astype(np.uint32)
    return Mesh(x, faces, object_of_vert=np.repeat(np.arange(2, dtype=np.uint32), [len(xa), len(xb)]), rest_x=x.copy())


@pytest.mark.parametrize("directions", [0, 1])
@pytest.mark.parametrize("length, axis", [(1, 0), (300, 0), (1000, 0), (2000, 1), (4000, 0), (4000, 2), (20000, 0)])
def test_both_forms_agree_on_long_edges(u26ctx, length, axis, directions):
    for seed in range(3):
        m = _mesh(length, seed, axis)
        got = []
        for form in (0, 1):
            sc = CollisionScene(u26ctx, m)
            sc.construct_lbvh()
            got.append(sc.untangle_pass(prp_params(max_contours=64, form=form, direction_mode=directions)))
            sc.close()
        batched, plain = got
        assert len(plain.hits) > 0 and sum(len(h) for h in plain.hits) > 0
        assert [len(h) for h in batched.hits] == [len(h) for h in plain.hits]
        for a, b in zip(batched.hits, plain.hits):
            assert a.tobytes() == b.tobytes()
        assert batched.results.tobytes() == plain.results.tobytes()
    assert u26ctx.device_errors() == 0


@pytest.mark.parametrize("length, directions, seed, rechecks, flips", [
    (1, 1, 0, 5560, 32), (300, 1, 1, 32352, 282), (1000, 0, 2, 7848, 36), (1000, 1, 1, 43429, 288), (4000, 0, 1, 19002, 21),
    (4000, 1, 2, 49957, 149), (20000, 0, 2, 65730, 24), (20000, 1, 0, 187364, 183)])
def test_recheck_counts_on_long_edges(u26ctx, length, directions, seed, rechecks, flips):
    """The counted FP64 rechecks are those of the leaf tests that a walk testing the boxes' bounds themselves makes
    (its counts are given), not of what the margins on centres and half extents add."""
    sc = CollisionScene(u26ctx, _mesh(length, seed, 0))
    sc.construct_lbvh()
    res = sc.untangle_pass(prp_params(max_contours=64, direction_mode=directions, fp64_recheck=1))
    sc.close()
    assert (res.fp64["rechecks"], res.fp64["flips"]) == (rechecks, flips)
