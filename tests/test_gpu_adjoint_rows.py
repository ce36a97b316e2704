"""Gradient rows of segments whose samples leave their brick's slot: the brick
step of the uniforms is the caller's, and a step of several texels carries the
later samples of a segment into neighbouring slots.  The samples that stay in
the slot have to keep its row, whatever the others before them looked up.
Against the oracle's binary64 adjoint, per texel within 1e-3 relative plus 1e-5
times the texel's sum of term magnitudes (the bound of the other adjoint
checks), in dense rows and in rows claimed by the touched slots."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", ["dense", "sparse"])
@pytest.mark.parametrize("form", [{}, {"f64": True}, {"warp_sum": True}, {"spread": True}])
@pytest.mark.parametrize("step", [(4.0, 4.0, 4.0), (2.5, -3.0, 1.0)])
def test_samples_out_of_the_slot(rows, form, step):
    sc = helpers.Scene(seed=2, depth=4, fmt="fp32")
    g = helpers.GpuScene(sc)
    pool = sc.pool.copy()
    pool.view(np.float32).reshape(-1, 4)[:, 3] *= 0.05  # rays that cross many bricks
    g.ctx.upload_bricks(np.arange(pool.shape[0], dtype=np.uint32), pool)
    u = sc.uniforms(sc.view(5, 61, 40))
    for a in range(3):
        u.brick_step_vector[a] *= step[a]
    H, W, n = u.height, u.width, pool.shape[0]
    ck = torch.empty(vv.Context.ckpt_bytes(W, H, 16), dtype=torch.uint8, device="cuda")
    g.ctx.forward_ckpt(u, 0, ck.data_ptr(), 16)
    dl = np.random.default_rng(7).standard_normal((H, W, 4)).astype(np.float32)
    dl_t = torch.from_numpy(dl).cuda()
    grad = torch.zeros((n, 1000, 4), dtype=torch.float64 if form.get("f64") else torch.float32, device="cuda")
    smap = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    used = torch.zeros(1, dtype=torch.int32, device="cuda")
    kw = dict(slot_map=smap.data_ptr(), rows_used=used.data_ptr(), rows_cap=n) if rows == "sparse" else {}
    g.ctx.backward_ex(u, dl_t.data_ptr(), ck.data_ptr(), 16, grad.data_ptr(), **form, **kw)
    g.ctx.synchronize()
    assert g.ctx.device_status() == 0
    got = grad.cpu().numpy().astype(np.float64)
    if rows == "sparse":
        m = smap.cpu().numpy()
        claimed, got = got, np.zeros_like(got)
        got[m >= 0] = claimed[m[m >= 0]]
    mag = np.zeros((n, 1000, 4))
    ref = go.backward(u, sc.oracle_scene(pool), dl, grad_abs=mag)
    assert np.abs(ref).max() > 0
    assert (np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5 * mag).all()
