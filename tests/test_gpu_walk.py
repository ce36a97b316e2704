"""The unit-box walk's dispatch and its rare paths against the FP32 oracle:
volume boxes other than [0,1]^3 (walked from the words), child pointers that
are not at a block's corner or leave the grid, trees deeper than the kept
path, frames that end inside a warp's tile, and sparse bricks that a ray
steps over by the projections of their occupied cells.  Usage lists, masks
and requests bit-exact; colour equal (both sides run the same binary32
operations)."""
import numpy as np
import pytest

import voxviz_b200 as vv
from oracle import gv_oracle as go
from tests import helpers

pytestmark = pytest.mark.gpu

RESIDENT, CONSTANT = 0x80000000, 0x40000000


def draw(words, pool, slots, u, fmt="rgba8"):
    ctx = vv.Context(0)
    ctx.upload_nodes(words)
    ctx.create_brickpool(slots, fmt)
    ctx.upload_bricks(np.arange(pool.shape[0], dtype=np.uint32), pool)
    jit = vv.make_jitter(7)
    ctx.set_jitter(jit)
    sc = helpers.GpuScene.__new__(helpers.GpuScene)
    sc.ctx = ctx
    return sc.render(u), helpers.oracle_frame(u, go.Scene(words, pool, slots, vv.fmt_code(fmt), jit))


def same(got, ref):
    assert got["status"] == ref["status"]
    assert np.array_equal(got["usage"], ref["usage"])
    assert np.array_equal(got["mask"], ref["mask"])
    assert np.array_equal(got["requests"], ref["requests"])
    assert np.array_equal(got["color"], ref["color"])


@pytest.mark.parametrize("lo,hi", [((0.0, 0.0, 0.0), (1.0, 1.0, 0.75)), ((0.125, 0.0, 0.0), (1.0, 0.875, 1.0)),
                                   ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0))])
@pytest.mark.parametrize("size", [(64, 48), (37, 29), (1, 1), (9, 5)])
def test_boxes_and_ragged_frames(lo, hi, size):
    sc = helpers.Scene(seed=1, depth=4, fmt="rgba8")
    u = sc.uniforms(sc.view(3, *size))
    u.vol_extent_min[:] = lo
    u.vol_extent_max[:] = hi
    same(*draw(sc.words, sc.pool, sc.slots, u))


def chain_tree(depth, dims, step, first):
    """Nodes on a chain: every level has one child that goes on (the corner of
    its block nearest the origin), the others are transparent constants; the
    deepest holds a brick.  Blocks at `first` + level * step along x."""
    dx, dy, dz = dims
    words = np.zeros((dz, dy, dx, 2), dtype=np.uint32)
    words[..., 0] = CONSTANT
    at = (0, 0, 0)
    for level in range(depth):
        b = (first + level * step, 0, 0)
        words[at[2], at[1], at[0], 0] = CONSTANT | (b[0] << 20) | (b[1] << 10) | b[2]
        at = b
    words[at[2], at[1], at[0]] = (RESIDENT, (1 << 20) | (1 << 10) | 1)
    return words


@pytest.mark.parametrize("depth,step,first,dims", [
    (3, 2, 2, (10, 2, 2)),      # blocks at their corners
    (3, 3, 1, (12, 2, 2)),      # odd pointers: children in two blocks
    (3, 4, 6, (10, 2, 2)),      # the second pointer leaves the grid
    (13, 2, 2, (40, 2, 2)),     # deeper than the kept path
])
def test_pointers_and_depths(depth, step, first, dims):
    rng = np.random.default_rng(depth)
    words = chain_tree(depth, dims, step, first) if first + (depth - 1) * step < dims[0] else None
    if words is None:  # the pointer out of the grid: the chain ends there
        words = chain_tree(1, dims, step, first)
        words[0, 0, first, 0] = CONSTANT | ((first + step) << 20)
    pool = rng.integers(1, 120, size=(8, 4000), dtype=np.uint8)
    sc = helpers.Scene(seed=1, depth=3, fmt="rgba8")
    look, up = vv.look_at((-0.05, -0.08, -0.06), (0.02, 0.03, 0.025))
    cam = vv.make_camera((-0.05, -0.08, -0.06), look, up, 48, 40, near=0.01)
    u = vv.compute_uniforms(sc.octree.info, cam, (2, 2, 2), 1.0, 0.99)
    u.lod_scalar = 1e6  # no level of detail stops the descent
    u.max_segments = 4000
    same(*draw(words, pool, (2, 2, 2), u))


@pytest.mark.parametrize("fmt", ["rgba8", "fp16", "fp32"])
@pytest.mark.parametrize("keep", [0.0, 0.002, 0.02])
def test_sparse_bricks(fmt, keep):
    sc = helpers.Scene(seed=1, depth=4, fmt=fmt)
    rng = np.random.default_rng(5)
    tb = vv.TEXEL_BYTES[vv.fmt_code(fmt)]
    pool = sc.pool.copy().reshape(-1, 1000, tb)
    pool[rng.random(pool.shape[:2]) >= keep] = 0
    # single occupied corner texels too
    pool[::7] = 0
    pool[::7, 0] = sc.pool.reshape(-1, 1000, tb)[::7].max(axis=1)
    pool = np.ascontiguousarray(pool.reshape(pool.shape[0], -1))
    for seed in (3, 9):
        same(*draw(sc.words, pool, sc.slots, sc.uniforms(sc.view(seed, 160, 96)), fmt))
