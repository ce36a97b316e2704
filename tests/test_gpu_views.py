"""Launch forms chosen by size: rays per warp by the frame's pixels, and the
views of a differentiable call in one launch (16 a launch).  A frame on each
side of a line equals the FP32 oracle; the views' colours equal one view's
calls bit for bit, and their gradient the sum of the views' within the
rounding of its binary32 additions."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size", [(192, 128), (193, 128), (448, 256), (449, 256), (2, 2), (3, 5), (17, 9)])
@pytest.mark.parametrize("lit", [False, True])
def test_rays_per_warp(size, lit):
    sc = helpers.Scene(seed=1, depth=4, fmt="rgba8")
    g = helpers.GpuScene(sc)
    u = sc.uniforms(sc.view(3, *size))
    grads = None
    if lit:
        n = sc.xyz.shape[0]
        grads = np.zeros((sc.pool.shape[0], vv.BRICK_BYTES[vv.fmt_code("fp32")]), dtype=np.uint8)
        grads[:n] = sc.octree.produce_gradients(sc.xyz, "fp32")
        g.ctx.create_gradpool("fp32")
        g.ctx.upload_gradients(np.arange(n, dtype=np.uint32), grads[:n])
        u.compute_lighting = 1
    got = g.render(u)
    ref = helpers.oracle_frame(u, go.Scene(sc.words, sc.pool, sc.slots, sc.fmt, sc.jitter, grads=grads,
                                           grad_fmt=vv.fmt_code("fp32")))
    assert got["status"] == ref["status"] == 0
    assert np.array_equal(got["usage"], ref["usage"]) and np.array_equal(got["requests"], ref["requests"])
    assert np.abs(got["color"] - ref["color"]).max() <= 1.0 / 255.0


@pytest.mark.parametrize("fmt,n,size", [("fp32", 1, (33, 21)), ("fp32", 2, (33, 21)), ("rgba8", 17, (33, 21)),
                                        ("fp16", 3, (131, 97)), ("fp32", 2, (257, 225))])
def test_views_of_one_call(fmt, n, size):
    sc = helpers.Scene(seed=1, depth=4, fmt=fmt)
    g = helpers.GpuScene(sc)
    W, H = size
    us = [sc.uniforms(sc.view(3 + v, W, H)) for v in range(n)]
    dev = torch.device("cuda", 0)
    nb = vv.Context.ckpt_bytes(W, H, 4)
    color = torch.zeros((n, H, W, 4), device=dev)
    ck = torch.zeros((n, nb), dtype=torch.uint8, device=dev)
    g.ctx.forward_ckpt_views(us, color.data_ptr(), ck.data_ptr(), 4)
    dl = torch.from_numpy(np.random.default_rng(n).standard_normal((n, H, W, 4)).astype(np.float32)).to(dev)
    slots = sc.pool.shape[0]
    grad = torch.zeros((slots, 1000, 4), device=dev)
    g.ctx.backward_views(us, dl.data_ptr(), ck.data_ptr(), 4, grad.data_ptr())
    one = torch.zeros((H, W, 4), device=dev)
    ref = torch.zeros((slots, 1000, 4), dtype=torch.float64, device=dev)
    for v, u in enumerate(us):
        g.ctx.forward_ckpt(u, one.data_ptr(), ck[0].data_ptr(), 4)
        assert torch.equal(one, color[v])
        g.ctx.backward_ex(u, dl[v].data_ptr(), ck[0].data_ptr(), 4, ref.data_ptr(), f64=True)
    torch.cuda.synchronize()
    assert g.ctx.device_status() == 0 and float(ref.abs().max()) > 0
    # binary32 sums of a few hundred terms of the texel's magnitude
    assert float((grad.double() - ref).abs().max()) <= 1e-4 * float(ref.abs().max())


def test_views_of_two_sizes_are_refused():
    sc = helpers.Scene(seed=1, depth=4, fmt="fp32")
    g = helpers.GpuScene(sc)
    us = [sc.uniforms(sc.view(3, 32, 16)), sc.uniforms(sc.view(4, 16, 32))]
    color = torch.zeros((2, 32, 16, 4), device="cuda")
    ck = torch.zeros(2 * vv.Context.ckpt_bytes(32, 16, 4), dtype=torch.uint8, device="cuda")
    with pytest.raises(vv.VVError):
        g.ctx.forward_ckpt_views(us, color.data_ptr(), ck.data_ptr(), 4)
