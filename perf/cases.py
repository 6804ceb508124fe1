"""The work that a program using this framework has it do, as measurable cases.

Six kinds, each through the entry points of the Python package:

* ``trees``   face and edge LBVH of a mesh constructed and refit (a solver's step start)
* ``refit``   both trees refit at new positions (every Newton iteration; swept for CCD)
* ``detect``  refit, fused edge-face detection, canonical order of the pairs
* ``narrow``  the same through the two-step interface: refit, broad-phase list, narrow phase, canonical order
* ``grad``    J and E over fixed supports with their gradients in positions and directions
* ``pass``    one untangling pass with its response pairs, as the command line's repair loop runs it

Meshes are this package's synthetic scenes: pairs of sheets, folded sheets, stacked layers,
batches of two-body scenes.
"""
import copy
import ctypes
import functools
import types

import numpy as np
import torch

from untangling26_b200 import _native as nat
from untangling26_b200 import synthetic
from untangling26_b200 import Context
from untangling26_b200.intersection_resolver import CollisionScene
from untangling26_b200.prp import EF_PAIR_DTYPE, HIT_DTYPE, RESULT_DTYPE, prp_params, response_params
from untangling26_b200.torch_ops import Support, objective


def listed():
    return [
        # step start of a coarse two-body scene, trees in the reference's topology (the drop-in default): launches and latency
        {"name": "trees_two_sheets32", "kind": "trees", "mesh": "two_sheets", "n": 32, "layers": 2, "parity": True},
        # step start of the self-colliding cloth (130,050 triangles)
        {"name": "trees_folded256", "kind": "trees", "mesh": "folded", "n": 256, "layers": 1, "parity": False},
        # step start of the largest scene: five stacked 512 x 512 sheets, 2.6 M triangles
        {"name": "trees_layers5x512", "kind": "trees", "mesh": "layers", "n": 512, "layers": 5, "parity": False},
        # a line search step's refit over the motion x_start -> x_end on the same scene
        {"name": "refit_layers5x512", "kind": "refit", "mesh": "layers", "n": 512, "layers": 5, "swept": True},
        # intersection check of a small scene: a handful of launches
        {"name": "detect_two_sheets64", "kind": "detect", "mesh": "two_sheets", "n": 64, "layers": 2},
        # intersection check of the largest scene (3.9 M edge queries)
        {"name": "detect_layers5x512", "kind": "detect", "mesh": "layers", "n": 512, "layers": 5},
        # the solver's own two call sites (broad-phase list, then narrow phase) on the folded cloth
        {"name": "narrow_folded256", "kind": "narrow", "mesh": "folded", "n": 256, "layers": 1},
        # differentiation: 32 x 32 sheets, 100 trials' size; then 128 x 128
        {"name": "grad_sheets32", "kind": "grad", "n": 32, "periods": 2},
        {"name": "grad_sheets128", "kind": "grad", "n": 128, "periods": 1},
        # repair pass of a small two-body scene, default settings
        {"name": "pass_two_sheets64", "kind": "pass", "mesh": "two_sheets", "n": 64, "layers": 2, "scenes": 0,
         "directions": 0, "opt": 0, "contours": 256, "solid": False},
        # repair pass of a folded cloth with the 26 directions and the refinement on S^2
        {"name": "pass_folded64_refined", "kind": "pass", "mesh": "folded", "n": 64, "layers": 1, "scenes": 0,
         "directions": 1, "opt": 4, "contours": 64, "solid": False},
        # sixteen independent two-body scenes as one batch
        {"name": "pass_batch16", "kind": "pass", "mesh": "batch", "n": 0, "layers": 0, "scenes": 16,
         "directions": 0, "opt": 0, "contours": 1 << 20, "solid": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("trees", "refit", "detect", "narrow", "grad", "pass"))
    if kind == "grad":
        return {"kind": "grad", "n": _log_int(rng, 24, 128), "periods": rng.randint(1, 3)}
    if kind == "pass":
        mesh = rng.choice(("two_sheets", "folded", "batch"))
        case = {"kind": "pass", "mesh": mesh, "n": 0, "layers": 0, "scenes": 0, "directions": 0, "opt": 0, "contours": 256,
                "solid": False}
        if mesh == "batch":
            return dict(case, scenes=rng.randint(2, 12), contours=1 << 20, solid=rng.random() < 0.3)
        if mesh == "two_sheets":
            return dict(case, n=_log_int(rng, 17, 97), layers=2, directions=rng.randint(0, 1), opt=rng.choice((0, 0, 1, 3)))
        return dict(case, n=_log_int(rng, 17, 64), layers=1, directions=rng.randint(0, 1), opt=rng.choice((0, 2, 4)), contours=64)
    mesh = rng.choice(("two_sheets", "folded", "layers"))
    case = {"kind": kind, "mesh": mesh}
    if mesh == "layers":
        case.update(layers=rng.randint(2, 5), n=_log_int(rng, 33, 511))
    else:
        case.update(layers=2 if mesh == "two_sheets" else 1, n=_log_int(rng, 9, 300))
    if kind == "trees":
        case["parity"] = rng.random() < 0.5
    if kind == "refit":
        case["swept"] = rng.random() < 0.5
    return case


# ---- inputs

@functools.lru_cache(maxsize=1)
def _context():
    return Context(0)


@functools.lru_cache(maxsize=4)
def _layer_topology(n, layers):
    """The stacked sheets' mesh (its tables depend on the sizes alone)."""
    return synthetic.layered_sheets(n, layers=layers, seed=0)


def _mesh(case, seed):
    """The case's mesh for `seed`: the same sizes, other shapes."""
    if case["mesh"] == "two_sheets":
        return synthetic.two_sheets(case["n"], seed=seed)
    if case["mesh"] == "folded":
        return synthetic.folded_sheet(case["n"], seed=seed)
    if case["mesh"] == "batch":
        m = synthetic.batch_scenes(case["scenes"], seed=seed)
        if case["solid"]:
            m.object_solid = np.ones(m.num_objects, np.uint32)
        return m
    # stacked layers 1 mm apart with seeded multi-octave waves of 2-20 mm
    m = copy.copy(_layer_topology(case["n"], case["layers"]))
    m.x = _layer_positions(case["n"], case["layers"], seed)
    return m


def _layer_positions(n, layers, seed):
    rng = np.random.default_rng(seed)
    u = np.linspace(0.0, 1.0, n)
    h = 1.0 / (n - 1)
    out = np.empty((layers, n, n, 3), np.float32)
    for k in range(layers):
        shift = rng.uniform(0.2, 0.45, 2) * h * (k > 0)
        z = np.zeros((n, n))
        for o in range(4):
            for _ in range(3):
                f = rng.uniform(-1.0, 1.0, 2) * 2 ** (o + 1)
                z += 0.5 ** o * np.outer(np.sin(2 * np.pi * (f[0] * u + rng.uniform())), np.sin(2 * np.pi * (f[1] * u + rng.uniform())))
        out[k, :, :, 0] = (u + shift[0])[:, None]
        out[k, :, :, 1] = (u + shift[1])[None, :]
        out[k, :, :, 2] = 0.001 * k + rng.uniform(0.002, 0.020) * z / np.abs(z).max()
    return out.reshape(-1, 3)


def _moved(x, n, seed):
    """End positions of a step: every vertex moved by up to a tenth of an edge length."""
    rng = np.random.default_rng(seed + 1)
    return (x + rng.uniform(-0.1, 0.1, x.shape) / n).astype(np.float32)


class _Words:
    """Device memory of the library as an array; `owner` lives as long as a tensor made of it."""

    def __init__(self, p, shape, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (int(p), False), "version": 3, "strides": None}


def _tree_arrays(scene, tree):
    """The tree's device arrays, as the solver's kernels read them (no copies)."""
    a = nat.U26LbvhArrays()
    scene.ctx.check(scene.ctx.lib.u26_lbvh_arrays_get(tree.handle, ctypes.byref(a)), "arrays_get")
    n, nn = a.num_leaves, a.num_nodes
    view = lambda p, shape, kind: torch.as_tensor(_Words(p, shape, kind, scene), device="cuda")  # noqa: E731
    return {
        "order": view(a.sorted_get_original, (n,), "<i4"),
        "codes": view(a.morton_sorted, (n,), "<i8"),
        "parent": view(a.parent, (nn,), "<i4"),
        "children": view(a.children, (nn, 2), "<i4"),
        "object": view(a.object_idx, (nn,), "<i4"),
        "boxes": view(a.node_aabb, (nn, 8), "<f4"),
    }


def prepare(case, seed):
    ctx = _context()
    if case["kind"] == "grad":
        g = _grad_inputs(case, seed)
        result = types.SimpleNamespace(hits=g["hits"], results=[{"dir": d} for d in g["dirs"]])
        mesh = types.SimpleNamespace(**{k: g[k] for k in ("rest_vert_area", "rest_edge_area", "rest_face_area", "vert_mass")})
        support = Support(ctx, result, mesh)
        x = torch.from_numpy(g["x"]).cuda().requires_grad_(True)
        dirs = torch.from_numpy(g["dirs"]).cuda().requires_grad_(True)
        return {"case": case, "support": support, "x": x, "dirs": dirs, "wJ": torch.from_numpy(g["wJ"]).cuda(),
                "wE": torch.from_numpy(g["wE"]).cuda()}
    mesh = _mesh(case, seed)
    # the broad-phase list of a folded cloth holds up to about 20 faces an edge
    scene = CollisionScene(ctx, mesh, d_hat=1e-3, thickness=0.0, max_broad_pairs=max(1 << 16, 40 * mesh.num_edges),
                           parity_tree=bool(case.get("parity", False)))
    state = {"case": case, "scene": scene}
    if case["kind"] != "trees":
        scene.construct_lbvh()
    if case["kind"] in ("trees", "refit"):
        state["face"] = _tree_arrays(scene, scene.face_tree)
        state["edge"] = _tree_arrays(scene, scene.edge_tree)
        state["x_end"] = torch.from_numpy(_moved(mesh.x, max(case["n"], 2), seed)).cuda() if case.get("swept") else scene.x
    if case["kind"] == "pass":
        state["params"] = prp_params(max_contours=case["contours"], batch_size=1 << 20 if case["mesh"] == "batch" else 32,
                                     direction_mode=case["directions"], opt_iterations=case["opt"])
        state["response"] = response_params()
        # the program's own arrays for the results, of sizes that the case's size bounds
        v, e, f = _sizes(case, most=True)
        pairs, hits, rows = (e // 4, v, 2) if case["mesh"] == "batch" else (e, 4 * v, 8)
        contours = 64 * max(case["scenes"], 8)
        state["out"] = {
            "pairs": np.zeros(pairs, EF_PAIR_DTYPE), "pair_indices": np.zeros((pairs, 2), np.uint32),
            "mesh_index": np.zeros(pairs, np.uint32), "contour_index": np.zeros(pairs, np.uint32),
            "pair_length": np.zeros(pairs, np.float32), "results": np.zeros(contours, RESULT_DTYPE),
            "hits": np.zeros(hits, HIT_DTYPE), "directions": np.zeros((26 * contours, 3), np.float32),
        }
        word = lambda *shape: torch.zeros(shape, dtype=torch.int32, device="cuda")  # noqa: E731
        state.update(narrow_list=word(hits, 16), narrow_indices=word(hits, 2),
                     vert_regions=word(rows * v), edge_regions=word(rows * e), face_regions=word(rows * f))
    return state


# ---- one pass

def run(state):
    kind = state["case"]["kind"]
    if kind == "grad":
        J, E = objective(state["x"], state["dirs"], state["support"])
        loss = (J * state["wJ"]).sum() + (E * state["wE"]).sum()
        gx, gr = torch.autograd.grad(loss, (state["x"], state["dirs"]))
        return {"J": J, "E": E, "x": gx, "dirs": gr}
    scene = state["scene"]
    if kind in ("trees", "refit"):
        if kind == "trees":
            scene.construct_lbvh()
        scene.face_tree.update_and_refit(scene.thickness, scene.x, state["x_end"], scene.faces)
        scene.edge_tree.update_and_refit(scene.thickness, scene.x, state["x_end"], scene.edges)
        if kind == "refit":
            return {"face": state["face"]["boxes"], "edge": state["edge"]["boxes"]}
        return {"face": state["face"], "edge": state["edge"]}
    if kind in ("detect", "narrow"):
        if kind == "detect":
            scene.detect_ef_fused()
        else:
            scene.broadphase_dcd_ef()
            scene.narrowphase_dcd_ef()
        n = scene.resolver.canonicalize(scene.mesh.num_edges, scene.mesh.num_faces)
        rows = scene.resolver.ef_list
        return {"count": n, "pairs": scene.resolver.ef_indices, "verts": rows[:, :5], "bary": rows.view(torch.float32)[:, 5:8]}
    r = scene.untangle_pass(state["params"], response=state["response"], narrow_list=state["narrow_list"],
                            narrow_indices=state["narrow_indices"])
    out, resp = state["out"], r.response
    if r.hits:
        np.concatenate(r.hits, out=out["hits"][:sum(len(h) for h in r.hits)])
    if r.directions:
        np.concatenate(r.directions, out=out["directions"][:sum(len(d) for d in r.directions)])
    for k in ("pairs", "pair_indices", "mesh_index", "contour_index", "pair_length", "results"):
        out[k][:len(getattr(r, k))] = getattr(r, k)
    for k in ("vert_regions", "edge_regions", "face_regions"):
        t = getattr(resp, k)
        state[k][:len(t)] = t
    words = {k: out[k].view(np.uint32).reshape(len(out[k]), -1) for k in ("pairs", "results", "hits")}
    floats = {k: w.view(np.float32) for k, w in words.items()}
    return {
        "counts": [len(r.pairs), len(r.results), sum(len(h) for h in r.hits), resp.num_pairs],
        "pair_verts": words["pairs"][:, :5], "pair_bary": floats["pairs"][:, 5:8], "pair_indices": out["pair_indices"],
        "mesh_index": out["mesh_index"], "contour_index": out["contour_index"], "pair_length": out["pair_length"],
        "results": words["results"][:, :24], "metrics": floats["results"][:, 24:35], "accepted": words["results"][:, 35],
        "hits": words["hits"][:, :9], "hit_values": floats["hits"][:, 9:], "directions": out["directions"],
        "response_verts": state["narrow_list"][:, :4], "response_values": state["narrow_list"].view(torch.float32)[:, 4:],
        "response_indices": state["narrow_indices"], **{k: state[k] for k in ("vert_regions", "edge_regions", "face_regions")},
    }


# ---- what a pass cannot do without

def _sizes(case, most=False):
    """(vertices, edges, faces) of the case's mesh (a batch: the expectation, or the most, of its draw)."""
    if case["kind"] == "grad":
        return 2 * case["n"] ** 2, 6 * case["n"] ** 2, 4 * case["n"] ** 2
    if case["mesh"] == "batch":
        f = (82000 if most else 31000) * case["scenes"]
        return f // 2 + 512, 3 * f // 2, f
    n, k = case["n"], case["layers"]
    return k * n * n, k * (3 * n * n - 4 * n + 1), 2 * k * (n - 1) ** 2


def work(case):
    v, e, f = _sizes(case)
    kind = case["kind"]
    if kind == "grad":
        hits = 5.2 * case["n"] ** 2  # the bumps cover almost the whole sheets; about one vertex, three edge and one face hit a vertex
        return {"bytes": 48 * hits + 12 * v * 2 + 4 * (v + e + f), "flops": 250 * hits}
    topology = lambda n: 4 * n + 8 * n + (4 + 8 + 4) * (2 * n - 1)  # order, codes, parent, children, object  # noqa: E731
    inputs = 16 * v + 12 * f + 8 * e
    boxes = 32 * (2 * f - 1) + 32 * (2 * e - 1)
    if kind == "trees":
        return {"bytes": inputs + boxes + topology(f) + topology(e), "flops": 30 * (e + f)}
    if kind == "refit":
        # both position arrays, the child links read, every box written
        return {"bytes": inputs + (12 * v if case["swept"] else 0) + 8 * (e + f) + boxes, "flops": 12 * (e + f)}
    if kind in ("detect", "narrow"):
        # the face tree refit (links read, boxes written), then read once with positions, edges and faces
        return {"bytes": inputs + 8 * f + 2 * 32 * (2 * f - 1) + 8 * v, "flops": 12 * f + 40 * e}
    # detection and both refits, the ray casts' trees read once
    return {"bytes": 2 * inputs + 2 * boxes + 16 * (e + f), "flops": 400 * (v + e + f) * (26 if case["directions"] else 8)}


# ---- 64-bit values

def _ef_exact(x, edges, faces):
    """Edge-face crossings in canonical order: barycentric time and face weights in 64 bits."""
    x = x.astype(np.float64)
    edges, faces = edges.astype(np.int64), faces.astype(np.int64)
    p, t = x[edges], x[faces]
    plo, phi, tlo, thi = p.min(1), p.max(1), t.min(1), t.max(1)
    cell = max((thi - tlo)[:, :2].max(), (phi - plo)[:, :2].max()) * 1.0001 + 1e-9
    base = x[:, :2].min(0) - 2 * cell
    width = int((x[:, 1].max() - base[1]) / cell) + 4
    tc = np.floor((tlo[:, :2] - base) / cell).astype(np.int64)
    tkey = tc[:, 0] * width + tc[:, 1]
    order = np.argsort(tkey, kind="stable")
    tkey = tkey[order]
    ec = np.floor((plo[:, :2] - base) / cell).astype(np.int64)
    found = []
    for di in (-1, 0, 1):
        for dj in (-1, 0, 1):
            key = (ec[:, 0] + di) * width + ec[:, 1] + dj
            a, b = np.searchsorted(tkey, key), np.searchsorted(tkey, key, side="right")
            cnt = b - a
            for s in range(0, len(key), 1 << 17):
                c = cnt[s:s + (1 << 17)]
                ei = np.repeat(np.arange(s, s + len(c)), c)
                fi = order[np.arange(len(ei)) - np.repeat(np.cumsum(c) - c, c) + np.repeat(a[s:s + len(c)], c)]
                near = ((plo[ei] <= thi[fi]) & (tlo[fi] <= phi[ei])).all(1)
                near &= ~(edges[ei][:, :, None] == faces[fi][:, None, :]).any((1, 2))
                found.append(np.stack([ei[near], fi[near]], 1))
    ef = np.concatenate(found)
    ef = ef[np.lexsort((ef[:, 1], ef[:, 0]))]
    p0, p1 = p[ef[:, 0], 0], p[ef[:, 0], 1]
    A, B, C = (t[ef[:, 1], k] for k in range(3))
    d = p1 - p0
    length = np.linalg.norm(d, axis=1)
    with np.errstate(all="ignore"):
        ray = d / length[:, None]
        N = np.cross(B - A, C - A)
        nlen = np.linalg.norm(N, axis=1)
        den = (-ray * N).sum(1)
        to = p0 - A
        s = (to * N).sum(1) / den
        cx = np.cross(-ray, to)
        u = ((C - A) * cx).sum(1) / den
        v = -((B - A) * cx).sum(1) / den
        time = s / length
        n = N / nlen[:, None]
        pen = np.minimum(np.abs(((p0 - A) * n).sum(1)), np.abs(((p1 - A) * n).sum(1)))
        keep = (length >= 1e-6) & (np.abs(den) >= nlen * 1e-6) & (s >= 0) & (s <= length)
        keep &= (np.minimum(np.minimum(u, v), 1 - u - v) >= 1e-4) & (np.minimum(time, 1 - time) >= 1e-4) & (pen >= 1e-4 * np.sqrt(nlen))
    return np.stack([1 - time, 1 - u - v, u], 1)[keep]


def _boxes_exact(codes, lo, hi):
    """Boxes of a binary radix tree over sorted unique codes, inner nodes first, rows of 8:
    minimum, 0, maximum, 1 (lo, hi: the leaves' boxes in sorted order)."""
    n = len(codes)
    i = np.arange(n - 1)

    def common(a, b):
        """Length of the common prefix of codes[a], codes[b] (-1 outside)."""
        ok = (b >= 0) & (b < n)
        z = codes[a] ^ codes[np.clip(b, 0, n - 1)]
        z_hi, z_lo = (z >> np.uint64(32)).astype(np.float64), (z & np.uint64(0xFFFFFFFF)).astype(np.float64)
        bits = np.where(z_hi > 0, 32 + np.frexp(z_hi)[1], np.where(z_lo > 0, np.frexp(z_lo)[1], 0))
        return np.where(ok, 64 - bits, -1)

    d = np.where(common(i, i + 1) > common(i, i - 1), 1, -1)
    d[0] = 1
    least = common(i, i - d)
    step = np.ones(n - 1, np.int64)
    step[:] = 1 << int(np.ceil(np.log2(n)))
    span = np.zeros(n - 1, np.int64)
    while step[0] >= 1:
        grow = common(i, i + (span + step) * d) > least
        span += step * grow
        step //= 2
    first, last = np.minimum(i, i + span * d), np.maximum(i, i + span * d)
    # range minima over powers of two
    k = np.frexp((last - first + 1).astype(np.float64))[1] - 1
    out = np.zeros((2 * n - 1, 8))
    out[:, 7] = 1.0
    v = np.concatenate([lo, -hi], 1)
    out[n - 1:, :3], out[n - 1:, 4:7] = lo, hi
    for q in range(int(k.max()) + 1):
        at = np.nonzero(k == q)[0]
        r = np.minimum(v[first[at]], v[last[at] - (1 << q) + 1])
        out[at, :3], out[at, 4:7] = r[:, :3], -r[:, 3:]
        w = 1 << q
        v = np.concatenate([np.minimum(v[:-w], v[w:]), v[-w:]]) if w < n else v
    return out


def _spread_bits(v):
    v = v.astype(np.uint64)
    out = np.zeros_like(v)
    for b in range(10):
        out |= ((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return out


def _tree_exact(x, end, prims, parity):
    """Boxes of one tree: leaves in the order of their 30-bit Morton codes (the codes are whole
    numbers that the 32-bit centres define), boxes in 64 bits."""
    k = prims.shape[1]
    P = x[prims.astype(np.int64)]
    third = np.float32(0.333333) if k == 3 else np.float32(0.5)
    total = (P[:, 0] + P[:, 1]) + P[:, 2] if k == 3 else P[:, 0] + P[:, 1]
    centre = third * total
    lo, hi = P.min(1), P.max(1)
    # the reference's global box covers the first ceil(vertices / 256) blocks of 256 primitives
    top = len(prims) if not parity else min(len(prims), 256 * -(-len(x) // 256))
    mn, mx = lo[:top].min(0), hi[:top].max(0)
    inv = np.float32(1.0) / np.maximum(mx - mn, np.float32(1e-6))
    q = np.clip((centre - mn) * inv * np.float32(1024.0), np.float32(0.0), np.float32(1023.0)).astype(np.uint32)
    code = (_spread_bits(q[:, 0]) << np.uint64(2)) | (_spread_bits(q[:, 1]) << np.uint64(1)) | _spread_bits(q[:, 2])
    code = (code << np.uint64(32)) | np.arange(len(prims), dtype=np.uint64)
    order = np.argsort(code, kind="stable")
    Q = end[prims.astype(np.int64)]
    lo, hi = np.minimum(lo, Q.min(1)).astype(np.float64), np.maximum(hi, Q.max(1)).astype(np.float64)
    return _boxes_exact(code[order], lo[order], hi[order])


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _grad_exact(_grad_inputs(case, seed))
    _, e, _ = _sizes(case)
    if kind == "pass" or e > (300_000 if kind in ("detect", "narrow") else 1_000_000):
        return None  # a pass is a sequence of decisions; the largest meshes take too long
    mesh = _mesh(case, seed)
    if kind in ("detect", "narrow"):
        bary = _ef_exact(mesh.x, mesh.edges, mesh.faces)
        rows = np.zeros((max(1 << 14, mesh.num_edges), 3))  # the list's capacity
        rows[:len(bary)] = bary
        return {"count": len(bary), "pairs": None, "verts": None, "bary": rows}
    end = _moved(mesh.x, max(case["n"], 2), seed) if case.get("swept") else mesh.x
    parity = bool(case.get("parity", False))
    face, edge = (_tree_exact(mesh.x, end, p, parity) for p in (mesh.faces, mesh.edges))
    if kind == "refit":
        return {"face": face, "edge": edge}
    rest = dict.fromkeys(("order", "codes", "parent", "children", "object"))
    return {"face": dict(rest, boxes=face), "edge": dict(rest, boxes=edge)}


# ---- supports of two crossing sheets, and J, E with their gradients in 64 bits

def _sheet_tables(n):
    """Faces, sorted unique edges (first, second vertex) and the id of the edge that starts at
    each vertex in each of the three directions (-1 where there is none) of one n x n sheet."""
    i, j = np.meshgrid(np.arange(n - 1), np.arange(n - 1), indexing="ij")
    v = (i * n + j).reshape(-1)
    faces = np.stack([np.stack([v, v + n, v + n + 1], 1), np.stack([v, v + n + 1, v + 1], 1)], 1).reshape(-1, 3)
    a = np.arange(n * n)
    r, c = a // n, a % n
    start, end, which = [], [], []
    for k, (di, dj) in enumerate(((0, 1), (1, 0), (1, 1))):
        ok = (r + di < n) & (c + dj < n)
        start.append(a[ok])
        end.append(a[ok] + di * n + dj)
        which.append(np.full(int(ok.sum()), k))
    start, end, which = map(np.concatenate, (start, end, which))
    order = np.lexsort((end, start))
    edges = np.stack([start, end], 1)[order]
    ids = np.full((n * n, 3), -1, np.int64)
    ids[edges[:, 0], which[order]] = np.arange(len(edges))
    return faces, edges, ids


def _cross2(a, b):
    return a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]


def _weights(p, a, b, c):
    """Barycentric weights of 2-D points p in triangles abc."""
    area = _cross2(b - a, c - a)
    w0, w1 = _cross2(b - p, c - p) / area, _cross2(c - p, a - p) / area
    return w0, w1, 1.0 - w0 - w1


def _grad_inputs(case, seed):
    """Two n x n sheets, B pushed through A in periods^2 bumps; per bump, the hits of B's part
    below A against A along a direction near +z: vertices of B on faces of A, edge pairs,
    vertices of A on faces of B."""
    n, periods = case["n"], case["periods"]
    rng = np.random.default_rng(seed)
    h = 1.0 / (n - 1)
    faces, edges, ids = _sheet_tables(n)
    r, c = np.divmod(np.arange(n * n), n)
    xa = np.stack([r * h, c * h, np.zeros(n * n)], 1)
    shift, amp = rng.uniform(0.2, 0.45, 2) * h, rng.uniform(0.05, 0.2)
    bump = np.sin(np.pi * periods * xa[:, 0]) ** 2 * np.sin(np.pi * periods * xa[:, 1]) ** 2
    xb = np.stack([xa[:, 0] + shift[0], xa[:, 1] + shift[1], 0.002 - amp * bump], 1)
    x = np.concatenate([xa, xb]).astype(np.float32)
    X = x.astype(np.float64)
    nv, ne, nf = n * n, len(edges), len(faces)
    region = np.minimum((xa[:, 0] * periods).astype(int), periods - 1) * periods + np.minimum((xa[:, 1] * periods).astype(int), periods - 1)
    below = X[nv:, 2] < -0.003
    hits, dirs = [], []
    for g in range(periods * periods):
        d = np.array([*rng.uniform(-0.08, 0.08, 2), 1.0])
        d = (d / np.linalg.norm(d)).astype(np.float32)
        D = d.astype(np.float64)
        # everything projected along d onto z = 0
        flat = X[:, :2] - X[:, 2:] * (D[:2] / D[2])
        fa, fb = flat[:nv], flat[nv:]
        vb = np.nonzero(below & (region == g))[0]
        if not len(vb):
            continue
        inside = np.zeros(nv, bool)
        inside[vb] = True
        out = []

        def put(kind, src, dst, sv, dv, b0, b1):
            rec = np.zeros(len(src), HIT_DTYPE)
            rec["type"], rec["src_id"], rec["dst_id"] = kind, src, dst
            rec["sv"][:, :sv.shape[1]], rec["dv"][:, :dv.shape[1]] = sv, dv
            rec["bary"][:, 0], rec["bary"][:, 1] = b0, b1
            out.append(rec)

        # vertices of B on faces of A (a regular grid)
        q = fb[vb] / h
        cell = np.clip(np.floor(q).astype(int), 0, n - 2)
        f = q - cell
        face = 2 * (cell[:, 0] * (n - 1) + cell[:, 1]) + (f[:, 1] > f[:, 0])
        tri = faces[face]
        w0, w1, w2 = _weights(fb[vb], fa[tri[:, 0]], fa[tri[:, 1]], fa[tri[:, 2]])
        ok = np.minimum(np.minimum(w0, w1), w2) > 1e-6
        put(0, nv + vb[ok], face[ok], (nv + vb)[ok, None], tri[ok], w0[ok], w1[ok])
        # edges of B on edges of A: the 5 x 5 vertices around B's start, three edges at each
        be = np.nonzero(inside[edges].all(1))[0]
        p0, p1 = fb[edges[be, 0]], fb[edges[be, 1]]
        near = np.floor(np.minimum(p0, p1) / h).astype(int)
        for oi in range(-1, 3):
            for oj in range(-1, 3):
                at = near + (oi, oj)
                okv = (at >= 0).all(1) & (at < n).all(1)
                vid = np.where(okv, at[:, 0] * n + at[:, 1], 0)
                for k in range(3):
                    eid = np.where(okv, ids[vid, k], -1)
                    m = np.nonzero(eid >= 0)[0]
                    ae = edges[eid[m]]
                    q0, q1 = fa[ae[:, 0]], fa[ae[:, 1]]
                    u, w = p1[m] - p0[m], q1 - q0
                    det = _cross2(u, w)
                    with np.errstate(all="ignore"):
                        s, t = _cross2(q0 - p0[m], w) / det, _cross2(q0 - p0[m], u) / det
                        ok = (np.abs(det) > 0.2 * h * h) & (np.minimum(np.minimum(s, 1 - s), np.minimum(t, 1 - t)) > 1e-3)
                    if ok.any():
                        # bary: weights of each edge's first vertex
                        put(1, ne + be[m][ok], eid[m][ok], nv + edges[be[m][ok]], ae[ok], (1 - s)[ok], (1 - t)[ok])
        # vertices of A on faces of B around them
        bf = np.nonzero(inside[faces].all(1))[0]
        tri = faces[bf]
        T = [fb[tri[:, k]] for k in range(3)]
        lo = np.ceil(np.minimum(np.minimum(T[0], T[1]), T[2]) / h).astype(int)
        for oi in range(3):
            for oj in range(3):
                at = lo + (oi, oj)
                okv = (at >= 0).all(1) & (at < n).all(1)
                vid = np.where(okv, at[:, 0] * n + at[:, 1], 0)
                w0, w1, w2 = _weights(fa[vid], *T)
                ok = okv & (np.minimum(np.minimum(w0, w1), w2) > 1e-6)
                put(2, nf + bf[ok], vid[ok], nv + tri[ok], vid[ok, None], w0[ok], w1[ok])
        rec = np.concatenate(out)
        hits.append(rec[np.lexsort((rec["dst_id"], rec["src_id"], rec["type"]))])
        dirs.append(d)
    area = 0.5 * h * h
    face_area = np.full(2 * nf, area)
    vert_area = np.concatenate([np.bincount(faces.reshape(-1), minlength=nv) * area / 3.0] * 2)
    around = np.sort(np.concatenate([faces[:, [0, 1]], faces[:, [1, 2]], faces[:, [0, 2]]]), 1)
    eid = np.searchsorted(edges[:, 0] * nv + edges[:, 1], around[:, 0] * nv + around[:, 1])
    edge_area = np.concatenate([np.bincount(eid, minlength=ne) * area / 3.0] * 2)
    f32 = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    return {"x": x, "dirs": np.stack(dirs), "hits": hits, "rest_vert_area": f32(vert_area), "rest_edge_area": f32(edge_area),
            "rest_face_area": f32(face_area), "vert_mass": f32(vert_area * 0.2),
            "wJ": f32(rng.uniform(0.5, 2.0, len(hits))), "wE": f32(rng.uniform(0.5, 2.0, len(hits)))}


def _deepest(h, x, d):
    """The hit that 32-bit depths make the deepest (the first of equals)."""
    dot = lambda a, b: (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]) + a[..., 2] * b[..., 2]  # noqa: E731
    cross = lambda a, b: np.stack([a[:, (k + 1) % 3] * b[:, (k + 2) % 3] - a[:, (k + 2) % 3] * b[:, (k + 1) % 3]  # noqa: E731
                                   for k in range(3)], 1)
    s, t = x[h["sv"]], x[h["dv"]]
    kind = h["type"][:, None]
    tri = np.where(kind[:, :, None] == 2, s, t)
    n = np.where(kind == 1, cross(s[:, 1] - s[:, 0], t[:, 1] - t[:, 0]), cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]))
    return int((dot(t[:, 0] - s[:, 0], n) / dot(d, n)).argmax())


def _grad_exact(g):
    x = torch.from_numpy(g["x"].astype(np.float64)).requires_grad_(True)
    dirs = torch.from_numpy(g["dirs"].astype(np.float64)).requires_grad_(True)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a).astype(np.float64))  # noqa: E731
    area = [t(g["rest_vert_area"]), t(g["rest_edge_area"]), t(g["rest_face_area"])]
    inv_mass = 1.0 / torch.clamp(t(g["vert_mass"]), min=1e-8)
    J, E = [], []
    for c, h in enumerate(g["hits"]):
        A, delta, kappa = [], [], []
        for kind in range(3):
            q = h[h["type"] == kind]
            sv, dv = torch.from_numpy(q["sv"].astype(np.int64)), torch.from_numpy(q["dv"].astype(np.int64))
            b0, b1 = t(q["bary"][:, 0]), t(q["bary"][:, 1])
            A.append(area[kind][torch.from_numpy(q["src_id"].astype(np.int64))])
            if kind == 1:
                s, d = x[sv[:, :2]], x[dv[:, :2]]
                n, w = torch.linalg.cross(s[:, 1] - s[:, 0], d[:, 1] - d[:, 0]), d[:, 0] - s[:, 0]
                ms, md = inv_mass[sv[:, :2]], inv_mass[dv[:, :2]]
                kappa.append(b0 ** 2 * ms[:, 0] + (1 - b0) ** 2 * ms[:, 1] + b1 ** 2 * md[:, 0] + (1 - b1) ** 2 * md[:, 1])
            else:
                tri, p = (x[dv], x[sv[:, 0]]) if kind == 0 else (x[sv], x[dv[:, 0]])
                m, mp = (inv_mass[dv], inv_mass[sv[:, 0]]) if kind == 0 else (inv_mass[sv], inv_mass[dv[:, 0]])
                n = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
                w = tri[:, 0] - p if kind == 0 else p - tri[:, 0]
                kappa.append(mp + b0 ** 2 * m[:, 0] + b1 ** 2 * m[:, 1] + (1 - b0 - b1) ** 2 * m[:, 2])
            delta.append((w * n).sum(1) / (n @ dirs[c]))
        A, delta, kappa = torch.cat(A), torch.cat(delta), torch.cat(kappa)
        J.append(A.sum() * delta[_deepest(h, g["x"], g["dirs"][c])] ** 2)
        E.append(((delta + 3e-3) ** 2 / kappa).sum())
    J, E = torch.stack(J), torch.stack(E)
    gx, gr = torch.autograd.grad((J * t(g["wJ"])).sum() + (E * t(g["wE"])).sum(), (x, dirs))
    return {"J": J.detach(), "E": E.detach(), "x": gx, "dirs": gr}
