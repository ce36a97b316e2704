"""The forms of a launch give the same pixels and the same gradient.

Frames: 4, 16 or 32 rays a warp by the frame's pixels.  A frame with a smaller
width and height and the same ray generation is a crop of the larger one, so
crops on each side of the lines equal it bit for bit, in every format and lit.

Views of a differentiable call: plain atomics take up to 16 views a launch,
binary64 and warp-summed rows a launch a view, spread copies are shared by the
views and sparse rows claimed by all of them.  Each against the oracle's
binary64 adjoint, per texel within 1e-3 relative plus 1e-5 times the texel's
sum of term magnitudes."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fmt,lit", [("rgba8", False), ("fp16", False), ("fp32", False), ("dxt5", False), ("rgba8", True),
                                     ("fp32", True)])
def test_crops_of_a_frame(fmt, lit):
    sc = helpers.Scene(seed=1, depth=4, fmt=fmt)
    g = helpers.GpuScene(sc)
    u = sc.uniforms(sc.view(3, 449, 257))
    if lit:
        n = sc.xyz.shape[0]
        g.ctx.create_gradpool("fp32")
        g.ctx.upload_gradients(np.arange(n, dtype=np.uint32), sc.octree.produce_gradients(sc.xyz, "fp32"))
        u.compute_lighting = 1
    whole = g.render(u, passes=vv.VV_PASS_RAYCAST)
    assert whole["status"] == 0 and whole["color"].max() > 0
    for w, h in ((449, 255), (448, 256), (331, 75), (193, 128), (192, 128), (97, 131), (31, 5)):
        u.width, u.height = w, h
        crop = g.render(u, passes=vv.VV_PASS_RAYCAST)
        assert np.array_equal(crop["color"], whole["color"][:h, :w])
        assert np.array_equal(crop["usage"], whole["usage"][:h, :w])


@pytest.mark.parametrize("rows", ["dense", "sparse"])
@pytest.mark.parametrize("form", [{}, {"spread": True}, {"f64": True}, {"warp_sum": True},
                                  {"warp_sum": True, "spread": True}, {"warp_sum": True, "f64": True}])
@pytest.mark.parametrize("n,size", [(3, (33, 21)), (18, (19, 13))])
def test_views_of_a_call(rows, form, n, size):
    sc = helpers.Scene(seed=1, depth=4, fmt="fp32")
    g = helpers.GpuScene(sc)
    W, H = size
    us = [sc.uniforms(sc.view(3 + v, W, H)) for v in range(n)]
    slots = sc.pool.shape[0]
    nb = vv.Context.ckpt_bytes(W, H, 4)
    ck = torch.zeros((n, nb), dtype=torch.uint8, device="cuda")
    dl = np.random.default_rng(n).standard_normal((n, H, W, 4)).astype(np.float32)
    dl_t = torch.from_numpy(dl).cuda()
    g.ctx.forward_ckpt_views(us, 0, ck.data_ptr(), 4)
    grad = torch.zeros((slots, 1000, 4), dtype=torch.float64 if form.get("f64") else torch.float32, device="cuda")
    smap = torch.full((slots,), -1, dtype=torch.int32, device="cuda")
    used = torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = dict(slot_map=smap.data_ptr(), rows_used=used.data_ptr(), rows_cap=slots) if rows == "sparse" else {}
    g.ctx.backward_views(us, dl_t.data_ptr(), ck.data_ptr(), 4, grad.data_ptr(), **form, **kw)
    g.ctx.synchronize()
    assert g.ctx.device_status() == 0
    got = grad.cpu().numpy().astype(np.float64)
    if rows == "sparse":
        m = smap.cpu().numpy()
        claimed, got = got, np.zeros_like(got)
        got[m >= 0] = claimed[m[m >= 0]]
    mag, ref = np.zeros((slots, 1000, 4)), np.zeros((slots, 1000, 4))
    for v in range(n):
        go.backward(us[v], sc.oracle_scene(), dl[v], grad=ref, grad_abs=mag)
    assert np.abs(ref).max() > 0
    assert (np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5 * mag).all()


@pytest.mark.parametrize("size", [(63, 47), (5, 3)])
@pytest.mark.parametrize("spread", [False, True])
def test_odd_frames_of_an_autograd_call(size, spread):
    from voxviz_b200 import diff
    sc = helpers.Scene(seed=1, depth=4, fmt="fp32")
    ctx = vv.Context(0)
    ctx.upload_nodes(sc.words)
    ctx.set_jitter(sc.jitter)
    pool = torch.from_numpy(np.ascontiguousarray(sc.pool).view(np.float32).reshape(-1, 1000, 4).copy()).cuda()
    pool.requires_grad_(True)
    W, H = size
    us = [sc.uniforms(sc.view(s, W, H)) for s in (3, 6)]
    dl = np.random.default_rng(W).standard_normal((2, H, W, 4)).astype(np.float32)
    img = diff.render(pool, ctx, sc.slots, us, 4, spread)
    got, = torch.autograd.grad(img, pool, torch.from_numpy(dl).cuda())
    assert diff.check_status(ctx) == 0
    mag, ref = np.zeros(tuple(pool.shape)), np.zeros(tuple(pool.shape))
    for v in range(2):
        go.backward(us[v], sc.oracle_scene(), dl[v], grad=ref, grad_abs=mag)
    got = got.cpu().numpy().astype(np.float64)
    assert np.abs(ref).max() > 0
    assert (np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5 * mag).all()


@pytest.mark.parametrize("form", [{}, {"f64": True}, {"warp_sum": True}, {"spread": True}])
@pytest.mark.parametrize("boxes,size", [("ubbuu", (33, 21)), ("b" * 18, (19, 13)), ("bu" * 3, (19, 13)), ("bb", (161, 157))])
def test_views_of_several_boxes(form, boxes, size):
    """Unit boxes (u) and others (b) in one call: each run of a kind is a launch."""
    sc = helpers.Scene(seed=1, depth=4, fmt="rgba8")
    g = helpers.GpuScene(sc)
    W, H = size
    n, slots = len(boxes), sc.pool.shape[0]
    us = [sc.uniforms(sc.view(3 + v, W, H)) for v in range(n)]
    for u, b in zip(us, boxes):
        if b == "b":
            u.vol_extent_max[2] = 0.75
    ck = torch.zeros((n, vv.Context.ckpt_bytes(W, H, 4)), dtype=torch.uint8, device="cuda")
    color = torch.zeros((n, H, W, 4), device="cuda")
    g.ctx.forward_ckpt_views(us, color.data_ptr(), ck.data_ptr(), 4)
    dl = np.random.default_rng(n).standard_normal((n, H, W, 4)).astype(np.float32)
    dl_t = torch.from_numpy(dl).cuda()
    grad = torch.zeros((slots, 1000, 4), dtype=torch.float64 if form.get("f64") else torch.float32, device="cuda")
    g.ctx.backward_views(us, dl_t.data_ptr(), ck.data_ptr(), 4, grad.data_ptr(), **form)
    g.ctx.synchronize()
    status = g.ctx.device_status(clear=True)  # (rays of a box may end at the iteration bound, as the oracle's do)
    mag, ref = np.zeros((slots, 1000, 4)), np.zeros((slots, 1000, 4))
    want = 0
    for v in range(n):
        frame = g.render(us[v], passes=vv.VV_PASS_RAYCAST)
        want = want or frame["status"]
        assert np.array_equal(color[v].cpu().numpy(), frame["color"])
        go.backward(us[v], sc.oracle_scene(), dl[v], grad=ref, grad_abs=mag)
    assert status == want
    got = grad.cpu().numpy().astype(np.float64)
    assert np.abs(ref).max() > 0
    assert (np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5 * mag).all()
