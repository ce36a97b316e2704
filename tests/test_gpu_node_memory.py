"""Device memory of node pools: the words and, memory allowing, as much again
for the walk's records, with a staging of 16 MB.  A pool whose records do not
fit is uploaded all the same and drawn from its words, in every form, with the
same results; patches and downloads work alike."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MB = 1 << 20


def padded(words, dims):
    """The same pool in a larger grid (the pointers are grid positions)."""
    big = np.zeros((dims[2], dims[1], dims[0], 2), dtype=np.uint32)
    z, y, x = words.shape[:3]
    big[:z, :y, :x] = words
    return big


def test_an_upload_takes_the_words_twice():
    sc = helpers.Scene(seed=1, depth=4, fmt="rgba8")
    words = padded(sc.words, (256, 256, 128))  # 64 MB
    ctx = vv.Context(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.upload_nodes(words)
    assert before - torch.cuda.mem_get_info()[0] <= 2 * words.nbytes + 20 * MB
    assert np.array_equal(ctx.download_nodes(), words)
    assert before - torch.cuda.mem_get_info()[0] <= 2 * words.nbytes + 20 * MB


def test_a_pool_without_room_for_its_records():
    sc = helpers.Scene(seed=2, depth=4, fmt="fp32")
    words = padded(sc.words, (256, 256, 128))
    ref = helpers.GpuScene(sc)
    g = helpers.GpuScene(sc)
    small = np.zeros((2, 2, 2, 2), dtype=np.uint32)
    g.ctx.upload_nodes(small)  # the words of before make room
    free = torch.cuda.mem_get_info()[0]
    room = words.nbytes + 40 * MB  # the words and the staging
    hog = [torch.empty(free - room, dtype=torch.uint8, device="cuda")]
    g.ctx.upload_nodes(words)
    del hog
    torch.cuda.empty_cache()
    assert np.array_equal(g.ctx.download_nodes(), words)
    u = sc.uniforms(sc.view(5, 61, 40))
    H, W = u.height, u.width
    a, b = g.render(u), ref.render(u)
    for k in ("color", "usage", "mask", "requests", "status"):
        assert np.array_equal(a[k], b[k]), k
    g.ctx.set_raycast_mode("refill")
    assert np.array_equal(g.render(u)["color"], b["color"])
    g.ctx.set_raycast_mode("tiles")
    color = torch.zeros((H, W, 4), device="cuda")
    vv.Batch(g.ctx, [(g.ctx, 0, u, color.data_ptr(), 0)]).render()
    torch.cuda.synchronize()
    assert np.array_equal(color.cpu().numpy(), b["color"])
    # forward and adjoint of two views
    us = [u, sc.uniforms(sc.view(6, W, H))]
    nb = vv.Context.ckpt_bytes(W, H, 4)
    color = torch.zeros((2, H, W, 4), device="cuda")
    ck = torch.zeros((2, nb), dtype=torch.uint8, device="cuda")
    dl = np.random.default_rng(1).standard_normal((2, H, W, 4)).astype(np.float32)
    dl_t = torch.from_numpy(dl).cuda()
    n = sc.pool.shape[0]
    grad = torch.zeros((n, 1000, 4), device="cuda")
    g.ctx.forward_ckpt_views(us, color.data_ptr(), ck.data_ptr(), 4)
    g.ctx.backward_views(us, dl_t.data_ptr(), ck.data_ptr(), 4, grad.data_ptr())
    g.ctx.synchronize()
    assert g.ctx.device_status() == 0
    mag = np.zeros((n, 1000, 4))
    want = np.zeros((n, 1000, 4))
    for v in range(2):
        assert np.array_equal(color[v].cpu().numpy(), ref.render(us[v])["color"])
        go.backward(us[v], sc.oracle_scene(), dl[v], grad=want, grad_abs=mag)
    got = grad.cpu().numpy().astype(np.float64)
    assert np.abs(want).max() > 0
    assert (np.abs(got - want) <= 1e-3 * np.abs(want) + 1e-5 * mag).all()
