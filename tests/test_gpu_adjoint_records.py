"""The adjoint's records (adjoint.cu): a ray with fewer sampled segments than
records replays each from its own, one with more walks from a point, and a
volume box other than [0,1]^3 walks from every record.  All against the
oracle's binary64 adjoint, per texel within 1e-3 relative plus 1e-5 times the
texel's sum of term magnitudes (the bound of the other adjoint checks); the
colour equals the plain draw's."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fmt", ["fp32", "rgba8"])
@pytest.mark.parametrize("per_ray", [1, 2, 3, 16])
@pytest.mark.parametrize("box", [(1.0, 1.0, 1.0), (1.0, 1.0, 0.75), (2.0, 2.0, 2.0)])
def test_records_match_fp64_oracle(fmt, per_ray, box):
    sc = helpers.Scene(seed=2, depth=4, fmt=fmt)
    g = helpers.GpuScene(sc)
    # an opacity low enough that rays cross many bricks
    pool = sc.pool.copy()
    if fmt == "fp32":
        f = pool.view(np.float32).reshape(-1, 4)
        f[:, 3] *= 0.05
    else:
        pool.reshape(-1, 4)[:, 3] = (pool.reshape(-1, 4)[:, 3] * 0.05).astype(np.uint8)
    g.ctx.upload_bricks(np.arange(pool.shape[0], dtype=np.uint32), pool)
    u = sc.uniforms(sc.view(5, 61, 40))
    u.vol_extent_max[:] = box
    H, W = u.height, u.width
    color = torch.zeros((H, W, 4), dtype=torch.float32, device="cuda")
    ck = torch.empty(vv.Context.ckpt_bytes(W, H, per_ray), dtype=torch.uint8, device="cuda")
    g.ctx.forward_ckpt(u, color.data_ptr(), ck.data_ptr(), per_ray)
    assert np.array_equal(color.cpu().numpy(), g.render(u, passes=vv.VV_PASS_RAYCAST)["color"])
    dl = np.random.default_rng(per_ray).standard_normal((H, W, 4)).astype(np.float32)
    dl_t = torch.from_numpy(dl).cuda()
    grad = torch.zeros((pool.shape[0], 1000, 4), dtype=torch.float32, device="cuda")
    g.ctx.backward(u, dl_t.data_ptr(), ck.data_ptr(), per_ray, grad.data_ptr())
    g.ctx.synchronize()
    assert g.ctx.device_status() == 0
    mag = np.zeros((pool.shape[0], 1000, 4))
    ref = go.backward(u, sc.oracle_scene(pool), dl, grad_abs=mag)
    got = grad.cpu().numpy().astype(np.float64)
    assert np.abs(ref).max() > 0
    assert (np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5 * mag).all()
