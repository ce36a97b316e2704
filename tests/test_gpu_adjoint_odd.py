"""Frames of an odd number of pixels: a view's checkpoint records lie behind
8 bytes a pixel of headers and are 16-byte vectors, so the headers are rounded
up, in the buffer and in a view's share of a larger one."""
import numpy as np
import pytest

import voxviz_b200 as vv
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def fp32_scene():
    sc = helpers.Scene(seed=1, depth=5, fmt="fp32")
    return sc, helpers.GpuScene(sc)


@pytest.mark.parametrize("size", [(63, 47), (1, 1), (5, 3)])
@pytest.mark.parametrize("per_ray", [1, 16])
def test_odd_pixel_counts(fp32_scene, size, per_ray):
    from voxviz_b200 import diff
    sc, g = fp32_scene
    W, H = size
    u = sc.uniforms(sc.view(3, W, H))
    assert vv.Context.ckpt_bytes(W, H, per_ray) % 16 == 0
    ref = g.render(u, passes=vv.VV_PASS_RAYCAST)["color"]
    ctx = vv.Context(0)
    ctx.upload_nodes(sc.words)
    ctx.set_jitter(sc.jitter)
    pool = torch.from_numpy(np.ascontiguousarray(sc.pool).view(np.float32).reshape(-1, 1000, 4).copy()).cuda()
    pool.requires_grad_(True)
    img = diff.render(pool, ctx, sc.slots, [u, u], per_ray)
    (img ** 2).sum().backward()
    assert diff.check_status(ctx) == 0
    assert np.array_equal(img[0].detach().cpu().numpy(), ref) and torch.equal(img[0], img[1])
    assert torch.isfinite(pool.grad).all()
