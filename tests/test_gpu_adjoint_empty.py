"""Samples of empty cells after a transmittance that is not finite: an empty
cell adds nothing to the colour or the opacity, so the forward leaves both as
they are, and the adjoint's replay has to do the same (infinity times zero
would make every later sample's gradient a NaN).  A brick of a slab whose
opacities overflow, then empty texels, then another such slab (opacities of
one sign: the sums stay infinite)."""
import numpy as np
import pytest

import voxviz_b200 as vv
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

RESIDENT, CONSTANT = 0x80000000, 0x40000000
BRICK = (1 << 20) | (1 << 10) | 1


def overflowing_pool():
    pool = np.zeros((8, 10, 10, 10, 4), dtype=np.float32)
    pool[0, 0:3] = (1e-3, 1e-3, 1e-3, -1e30)
    pool[0, 7:10] = (0.5, 0.25, 0.125, -1e30)
    return pool


def words_of(levels):
    """The brick at the root, or at its eight children."""
    words = np.zeros((2, 2, 4, 2), dtype=np.uint32)
    words[0, 0, 0] = (RESIDENT, BRICK)
    if levels:
        words[0, 0, 0] = (CONSTANT | (2 << 20), 0)
        words[:, :, 2:4] = (RESIDENT, BRICK)
    return words


@pytest.mark.parametrize("levels,per_ray", [(0, 1), (0, 16), (1, 1), (1, 16)])
def test_empty_samples_keep_the_transmittance(levels, per_ray):
    sc = helpers.Scene(seed=1, depth=3, fmt="rgba8")
    eye = (0.45, 0.55, -0.3)
    look, up = vv.look_at(eye, (0.5, 0.5, 0.5))
    u = vv.compute_uniforms(sc.octree.info, vv.make_camera(eye, look, up, 24, 16, near=0.01), (2, 2, 2), 1.0, 0.99)
    u.lod_scalar = 1e6
    ctx = vv.Context(0)
    ctx.upload_nodes(words_of(levels))
    ctx.create_brickpool((2, 2, 2), "fp32")
    ctx.upload_bricks(np.arange(8, dtype=np.uint32), overflowing_pool().reshape(8, -1).view(np.uint8))
    ctx.set_jitter(sc.jitter)
    color = torch.zeros((16, 24, 4), device="cuda")
    ck = torch.empty(vv.Context.ckpt_bytes(24, 16, per_ray), dtype=torch.uint8, device="cuda")
    ctx.forward_ckpt(u, color.data_ptr(), ck.data_ptr(), per_ray)
    dl = torch.ones((16, 24, 4), device="cuda")
    dl[..., 3] = 0.0
    grad = torch.zeros((8, 10, 10, 10, 4), device="cuda")
    ctx.backward(u, dl.data_ptr(), ck.data_ptr(), per_ray, grad.data_ptr())
    ctx.synchronize()
    assert ctx.device_status() == 0
    rgb = color[..., :3]
    assert not torch.isnan(rgb).any() and torch.isposinf(rgb).any()
    # dL/d(rgb) is dL/dc times the weight and the transmittance: infinite in the far slab
    far = grad[0, 7:, ..., :3]
    assert not torch.isnan(far).any() and torch.isposinf(far).any()
