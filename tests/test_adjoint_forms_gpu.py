"""u26_prp_adjoint at the edges of its launch rule: contours of few hits are a warp's (up to 64 hits, 128 for 65 to 148
contours, more for very many), longer ones a cluster's; 16 and 17, 64 and 65, 148 and 149, 592 and 593, 2,368 and
more contours change the clusters' shape or make them loop. J and E are back-propagated together. The supports repeat a
few hits of a real pass, so the FP64 values follow from theirs (tolerance 2e-3 relative, the bar of the
fp32 kernel on real supports). Most of those hits are equally deep (flat sheets 2 mm apart): J's gradient is that
of the first hit of the largest fp32 depth."""
import types

import numpy as np
import pytest
import torch

from oracle import adjoint as adj
from test_adjoint_gpu import _support
from untangling26_b200.torch_ops import JFunction, Support

pytestmark = pytest.mark.gpu


def _base(ctx):
    """Up to seven hits of each type of a real support, and its direction."""
    m, res, _ = _support(ctx, 32, 0)
    c = int(np.argmax([len(h) for h in res.hits]))
    hits = res.hits[c]
    return m, np.concatenate([hits[hits["type"] == t][3::11][:7] for t in range(3)]), np.asarray(res.results[c]["dir"], np.float32)


def _depth32(h, x, r):
    """The kernel's depth: the same operations in the same order, in fp32."""
    dot = lambda a, b: (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]  # noqa: E731
    cross = lambda a, b: np.array([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]], np.float32)  # noqa: E731
    P = x[adj.hit_vertices(h)]
    if h["type"] == 1:
        n, w = cross(P[1] - P[0], P[3] - P[2]), P[2] - P[0]
    else:
        n, w = cross(P[2] - P[1], P[3] - P[1]), (P[1] - P[0] if h["type"] == 0 else P[0] - P[1])
    return dot(w, n) / dot(r, n)


def _lens(contours, *lens):
    return [lens[i * len(lens) // contours] if i % 3 else lens[i % len(lens)] for i in range(contours)]


@pytest.mark.parametrize("lens", [
    _lens(1, 64), _lens(1, 65), _lens(16, 0, 1, 64, 65, 9000), _lens(17, 63, 66, 2049), _lens(18, 8193, 1, 0, 33),
    _lens(64, 64, 65, 300), _lens(65, 1, 128, 129, 1025), _lens(148, 8, 128, 129, 4097), _lens(149, 64, 65, 0, 1100),
    _lens(592, 64, 65, 3), _lens(593, 1, 64, 65), _lens(2369, 64, 3, 148, 149), _lens(4200, 2, 33, 1024, 1025)], ids=lambda v: str(len(v)))
def test_adjoint_forms(u26ctx, lens):
    m, base, r = _base(u26ctx)
    result = types.SimpleNamespace(hits=[np.resize(base, n) for n in lens], results=[{"dir": r}] * len(lens))
    sup = Support(u26ctx, result, m)
    dev = torch.device("cuda", u26ctx.device)
    x = torch.from_numpy(m.x).to(dev).requires_grad_(True)
    dirs = sup.dirs.clone().requires_grad_(True)
    J, E = JFunction.apply(x, dirs, sup)
    wJ, wE = torch.linspace(2.0, 1.0, len(lens), device=dev), torch.linspace(0.5, 1.5, len(lens), device=dev)
    (J * wJ + E * wE).sum().backward()
    Jh, Eh, gx, gd = J.detach().cpu().numpy(), E.detach().cpu().numpy(), x.grad.cpu().numpy(), dirs.grad.cpu().numpy()
    x64, r64, mc = m.x.astype(np.float64), r.astype(np.float64), (m.rest_vert_area, m.rest_edge_area, m.rest_face_area, m.vert_mass)
    one = []
    for h in base:
        h1 = np.array([h], base.dtype)
        A1, d1 = adj.source_area(h, *mc[:3]), adj.delta(h, x64[adj.hit_vertices(h)], r64)
        _, E1, _ = adj.objective(h1, x64, r64, *mc)
        gJx, gJr, gEx, gEr = adj.gradients(h1, x64, r64, *mc)
        one.append((A1, d1, E1, gJx, gJr, gEx, gEr))
    depth = [_depth32(h, m.x, r) for h in base]
    assert depth.count(max(depth)) > 1
    gx_ref = np.zeros_like(x64)
    for i, n in enumerate(lens):
        times = [n // len(base) + (k < n % len(base)) for k in range(len(base))]
        A = sum(t * o[0] for t, o in zip(times, one))
        E64 = sum(t * o[2] for t, o in zip(times, one))
        present = [k for k, t in enumerate(times) if t]
        deep = max(present, key=lambda k: depth[k]) if present else -1
        D = one[deep][1] if present else 0.0
        assert abs(Jh[i] - A * D * D) <= 2e-3 * abs(A * D * D) and abs(Eh[i] - E64) <= 2e-3 * abs(E64)
        # the deepest hit's own gradient is that of A_h D^2
        a, b = float(wJ[i]) * (A / one[deep][0] if present else 0.0), float(wE[i])
        gr = sum(t * o[6] for t, o in zip(times, one)) * b + (a * one[deep][4] if present else 0.0)
        assert np.abs(gd[i] - gr).max() <= 2e-3 * np.abs(gr).max()
        gx_ref += sum(t * o[5] for t, o in zip(times, one)) * b + (a * one[deep][3] if present else 0.0)
    assert np.abs(gx - gx_ref).max() <= 2e-3 * np.abs(gx_ref).max()


@pytest.mark.parametrize("n, contours", [(1, 1), (40, 1), (64, 20), (65, 1), (700, 3), (9000, 2), (700, 20), (300, 200)])
def test_nan_depths(u26ctx, n, contours):
    """A hit of NaN depth is never the deepest, except as the support's first hit."""
    m, base, r = _base(u26ctx)
    # one vertex off the other hits' vertices
    verts = np.unique(np.concatenate([adj.hit_vertices(h) for h in base]))
    free = int(np.setdiff1d(np.arange(m.num_verts), verts)[0])
    bad = base[:1].copy()
    assert bad["type"][0] == 0
    bad["sv"][0, 0] = free
    x64, r64 = m.x.astype(np.float64), r.astype(np.float64)
    x = m.x.copy()
    x[free] = np.nan
    dev = torch.device("cuda", u26ctx.device)
    for at in (0, n // 2, n - 1):
        hits = np.resize(base, n)
        hits[at] = bad[0]
        result = types.SimpleNamespace(hits=[hits] * contours, results=[{"dir": r}] * contours)
        sup = Support(u26ctx, result, m)
        J, _ = JFunction.apply(torch.from_numpy(x).to(dev), sup.dirs, sup)
        J = J.cpu().numpy()
        if at == 0:
            assert np.isnan(J).all()
            continue
        A = sum(adj.source_area(h, m.rest_vert_area, m.rest_edge_area, m.rest_face_area) for h in hits)
        D = max(adj.delta(h, x64[adj.hit_vertices(h)], r64) for i, h in enumerate(hits[:len(base) + 1]) if i != at)
        if n > len(base) + 1:
            D = max(D, max(adj.delta(h, x64[adj.hit_vertices(h)], r64) for h in base))
        assert np.abs(J - A * D * D).max() <= 2e-3 * A * D * D
