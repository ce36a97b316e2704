"""Bricks far down a chain of nodes: one 2x2x2 block a level is all a chain
takes, so a pool holds chains of any depth.  The brick's depth sets the step
and the position in the brick, at depth 31 as at 32 and beyond.  A camera
inside the deepest node, at the scale of that node; against the FP32 oracle."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers
from tests.test_gpu_walk import chain_tree, draw, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [12, 23, 24, 31, 32, 33, 40])
@pytest.mark.parametrize("fmt", ["rgba8", "fp32"])
def test_brick_at_depth(depth, fmt):
    words = chain_tree(depth, (2 * depth + 4, 2, 2), 2, 2)
    rng = np.random.default_rng(depth)
    if fmt == "rgba8":
        pool = rng.integers(1, 60, size=(8, 4000), dtype=np.uint8)
    else:
        pool = rng.uniform(0.01, 0.2, size=(8, 4000)).astype(np.float32).view(np.uint8)
    sc = helpers.Scene(seed=1, depth=3, fmt=fmt)
    eye = (0.3, 0.4, 0.5)
    look, up = vv.look_at(eye, (0.9, 0.8, 0.7))
    u = vv.compute_uniforms(sc.octree.info, vv.make_camera(eye, look, up, 16, 8, near=0.01), (2, 2, 2), 1.0, 0.99)
    size = 2.0 ** -depth  # of the deepest node, which the camera is scaled into
    for a in range(3):
        u.camera_position[a] = eye[a] * size
        u.near_origin[a] *= size
        u.near_dx[a] *= size
        u.near_dy[a] *= size
    u.camera_inside = 1
    u.oct_tree_depth_minus_one = depth
    u.ray_step_size = size / 16.0
    u.pixel_size = -1.0  # no level of detail stops the descent
    u.max_segments = 20000
    got, ref = draw(words, pool, (2, 2, 2), u, fmt)
    assert ref["status"] == 0 and ref["color"].max() > 0
    same(got, ref)
