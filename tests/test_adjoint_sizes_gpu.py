"""u26_prp_adjoint at the edges of its launch rule: one, 18, 19, 148 and 149 contours, and supports of
no hit, one hit and around a warp, a block and a whole cluster of hits. The supports repeat a few
hits of a real pass, so the FP64 values are multiples of theirs (tolerance 2e-3 relative, the
bar of the fp32 kernel on real supports)."""
import types

import numpy as np
import pytest
import torch

from oracle import adjoint as adj
from test_adjoint_gpu import _support
from untangling26_b200.torch_ops import JFunction, Support

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[8193], [8192] + [0, 1, 31, 32, 33, 1023, 1024, 1025, 8191] * 2, [0] * 18 + [2049],
                                  [257] * 147 + [1], [0, 1, 255, 256, 257] * 30], ids=["1", "19", "19-last", "148", "150"])
def test_adjoint_support_sizes(u26ctx, lens):
    m, res, _ = _support(u26ctx, 32, 0)
    c = int(np.argmax([len(h) for h in res.hits]))
    hits = res.hits[c]
    # up to seven hits of each type
    base = np.concatenate([hits[hits["type"] == t][3::11][:7] for t in range(3)])
    r = np.asarray(res.results[c]["dir"], np.float32)
    result = types.SimpleNamespace(hits=[np.resize(base, n) for n in lens], results=[{"dir": r}] * len(lens))
    sup = Support(u26ctx, result, m)
    dev = torch.device("cuda", u26ctx.device)
    x = torch.from_numpy(m.x).to(dev).requires_grad_(True)
    dirs = sup.dirs.clone().requires_grad_(True)
    J, E = JFunction.apply(x, dirs, sup)
    w = torch.linspace(0.5, 1.5, len(lens), device=dev)
    (E * w).sum().backward()
    Jh, Eh, gx, gd = J.detach().cpu().numpy(), E.detach().cpu().numpy(), x.grad.cpu().numpy(), dirs.grad.cpu().numpy()
    x64, r64, mc = m.x.astype(np.float64), r.astype(np.float64), (m.rest_vert_area, m.rest_edge_area, m.rest_face_area, m.vert_mass)
    one = []
    for h in base:
        h1 = np.array([h], base.dtype)
        _, E1, _ = adj.objective(h1, x64, r64, *mc)
        _, _, gEx, gEr = adj.gradients(h1, x64, r64, *mc)
        one.append((adj.source_area(h, *mc[:3]), adj.delta(h, x64[adj.hit_vertices(h)], r64), E1, gEx, gEr))
    gx_ref = np.zeros_like(x64)
    for i, n in enumerate(lens):
        times = [n // len(base) + (k < n % len(base)) for k in range(len(base))]
        E64 = sum(t * o[2] for t, o in zip(times, one))
        D = max([o[1] for t, o in zip(times, one) if t], default=0.0)
        J64 = sum(t * o[0] for t, o in zip(times, one)) * D * D
        gr = sum(t * o[4] for t, o in zip(times, one)) * float(w[i])
        assert abs(Jh[i] - J64) <= 2e-3 * abs(J64) and abs(Eh[i] - E64) <= 2e-3 * abs(E64)
        assert np.abs(gd[i] - gr).max() <= 2e-3 * np.abs(gr).max()
        gx_ref += sum(t * o[3] for t, o in zip(times, one)) * float(w[i])
    assert np.abs(gx - gx_ref).max() <= 2e-3 * np.abs(gx_ref).max()
