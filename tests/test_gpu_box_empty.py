"""Empty cells in a volume box other than [0,1]^3: their samples are passed
over there too, in the draw, the checkpointing forward and the adjoint.  Seen by
what passing them over means for an infinite transmittance (as in
test_gpu_adjoint_empty): the colour and the far slab's gradient stay infinite
instead of becoming NaN."""
import numpy as np
import pytest

import voxviz_b200 as vv
from tests import helpers
from tests.test_gpu_adjoint_empty import overflowing_pool, words_of

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lo,hi", [((0.0, 0.0, 0.0), (1.0, 1.0, 0.9375)), ((0.125, 0.0, 0.0), (1.0, 0.875, 1.0))])
@pytest.mark.parametrize("form", [{}, {"f64": True}, {"warp_sum": True}])
def test_empty_samples_in_a_box(lo, hi, form):
    sc = helpers.Scene(seed=1, depth=3, fmt="rgba8")
    eye = (0.45, 0.55, -0.3)
    look, up = vv.look_at(eye, (0.5, 0.5, 0.5))
    u = vv.compute_uniforms(sc.octree.info, vv.make_camera(eye, look, up, 24, 16, near=0.01), (2, 2, 2), 1.0, 0.99)
    u.lod_scalar = 1e6
    u.vol_extent_min[:] = lo
    u.vol_extent_max[:] = hi
    ctx = vv.Context(0)
    ctx.upload_nodes(words_of(0))
    ctx.create_brickpool((2, 2, 2), "fp32")
    ctx.upload_bricks(np.arange(8, dtype=np.uint32), overflowing_pool().reshape(8, -1).view(np.uint8))
    ctx.set_jitter(sc.jitter)
    color, plain = (torch.zeros((16, 24, 4), device="cuda") for _ in range(2))
    ctx.render(u, color=plain.data_ptr(), passes=vv.VV_PASS_RAYCAST)
    ck = torch.empty(vv.Context.ckpt_bytes(24, 16, 4), dtype=torch.uint8, device="cuda")
    ctx.forward_ckpt(u, color.data_ptr(), ck.data_ptr(), 4)
    dl = torch.ones((16, 24, 4), device="cuda")
    dl[..., 3] = 0.0
    grad = torch.zeros((8, 10, 10, 10, 4), dtype=torch.float64 if form.get("f64") else torch.float32, device="cuda")
    ctx.backward_ex(u, dl.data_ptr(), ck.data_ptr(), 4, grad.data_ptr(), **form)
    ctx.synchronize()
    assert ctx.device_status() == 0
    assert torch.equal(color, plain)
    assert not torch.isnan(color[..., :3]).any() and torch.isposinf(color[..., :3]).any()
    far = grad[0, 7:, ..., :3]
    assert not torch.isnan(far).any() and torch.isposinf(far).any()
