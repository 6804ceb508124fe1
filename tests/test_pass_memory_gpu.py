"""Device memory that a pass of many hits takes: buffers sized to what a level asks for. The bound is what exact sizes
take (20.82 GB for 256 contours of the folded 256 x 256 sheet with 26 directions) and 2 %: about a hundred
allocations rounded up to 2 MB, and a growth slack of 32 MB on the few buffers that grow past it."""
import pytest
import torch

from untangling26_b200 import Context, synthetic
from untangling26_b200.intersection_resolver import CollisionScene
from untangling26_b200.prp import prp_params

pytestmark = pytest.mark.gpu


def test_pass_memory():
    ctx = Context(0)
    params = prp_params(max_contours=256, batch_size=256, direction_mode=1)
    # the kernels' own memory (local memory, modules) is the context's
    small = CollisionScene(ctx, synthetic.folded_sheet(32, seed=1))
    small.construct_lbvh()
    small.untangle_pass(params)
    small.close()
    m = synthetic.folded_sheet(256, seed=1)
    sc = CollisionScene(ctx, m)
    sc.construct_lbvh()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    res = sc.untangle_pass(params)
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    assert sum(len(h) for h in res.hits) > 0 and res.device_error_flags == 0
    assert taken <= 1.02 * 20.82e9
    sc.close()
    ctx.close()
