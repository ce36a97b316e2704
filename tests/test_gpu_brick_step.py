"""Brick steps that are no texel distances (infinite, NaN): a sample position
that is not finite reads the texels that clamping gives it, so a ray may not
pass a brick by the projections of its occupied cells.  Against the FP32
oracle, which reads every sample."""
import numpy as np
import pytest

import voxviz_b200 as vv
from tests import helpers
from tests.test_gpu_walk import draw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [np.nan, np.inf, -np.inf, 1e30])
@pytest.mark.parametrize("axis", [0, 2])
def test_steps_out_of_range(step, axis):
    sc = helpers.Scene(seed=1, depth=4, fmt="rgba8")
    pool = np.zeros_like(sc.pool)
    texels = pool.reshape(-1, 10, 10, 10, 4)  # z, y, x
    # only the first and the last texels along the axis: the middle of every brick is empty
    for at in (0, 9):
        (texels[:, :, :, at] if axis == 0 else texels[:, at])[...] = 9
    u = sc.uniforms(sc.view(3, 64, 48))
    u.brick_step_vector[axis] = step
    got, ref = draw(sc.words, pool, sc.slots, u)
    assert got["status"] == ref["status"]
    assert np.array_equal(got["usage"], ref["usage"])
    assert ref["color"].max() > 0
    assert np.array_equal(got["color"], ref["color"])
