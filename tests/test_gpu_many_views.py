"""A differentiable call of more views than 16 bits count: any number is taken,
16 a launch."""
import numpy as np
import pytest

import voxviz_b200 as vv
from tests import helpers

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_more_than_65536_views():
    from voxviz_b200 import diff
    sc = helpers.Scene(seed=1, depth=3, fmt="fp32")
    ctx = vv.Context(0)
    ctx.upload_nodes(sc.words)
    ctx.set_jitter(sc.jitter)
    pool = torch.from_numpy(np.ascontiguousarray(sc.pool).view(np.float32).reshape(-1, 1000, 4).copy()).cuda()
    pool.requires_grad_(True)
    a, b = (sc.uniforms(sc.view(s, 1, 1)) for s in (3, 5))
    n = 65537
    img = diff.render(pool, ctx, sc.slots, [a] * (n - 1) + [b], 2)
    two = diff.render(pool, ctx, sc.slots, [a, b], 2)
    assert torch.equal(img[:n - 1], two[:1].expand(n - 1, -1, -1, -1)) and torch.equal(img[n - 1], two[1])
    # the last view's gradient alone
    got, = torch.autograd.grad(img[n - 1].sum(), pool, retain_graph=True)
    ref, = torch.autograd.grad(two[1].sum(), pool)
    assert diff.check_status(ctx) == 0
    assert float(ref.abs().max()) > 0
    # one ray: each texel's sum has the same few terms in the same order but for the taps' rotation
    assert float((got - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
