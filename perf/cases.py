"""The measured workloads of the ray caster, through its public entry points.

Five kinds of call, over the sizes the repository's tests, benchmark and
configurations use:

* ``frame``   one draw of a resident octree (``Context.render``): the ray cast
  alone or with the selection mask, histopyramid and request compaction; every
  brick format, lit or not, cameras above the terrain or flying low in it;
* ``flight``  frames of a paged octree through the renderer plugin: draw,
  colour read-back and page-request service with an LRU pool that is smaller
  than the flight's bricks;
* ``batch``   many views of several octrees in one persistent launch;
* ``fit``     a step of fitting bricks to target views: the differentiable
  ray cast forward and backward through autograd (dense gradient);
* ``adjoint`` checkpointing forward and adjoint of one frame of a paged
  octree, the gradient in rows of the touched slots.

Every input follows from the case and the seed: the terrain, the cameras, the
noise of the targets.  ``exact`` restates the ray cast with plain tensors:
positions and decisions in binary32 in the order the shader is written, which
fixes the sample sequence, and filtering, compositing and the adjoint along
that sequence in binary64.
"""
import math

import numpy as np
import torch

import voxviz_b200 as vv
from voxviz_b200 import diff, scene

ALPHA_STOP = 0.99
JITTER_SEED = 7
PER_RAY = 16
TEXEL = {"rgba8": 4, "fp16": 8, "bf16": 8, "fp32": 16, "dxt5": 1.44}


def listed():
    return [
        # the smallest draw: a thumbnail of a small volume, where launches count
        {"name": "frame_thumbnail", "kind": "frame", "depth": 4, "width": 96, "height": 64, "fmt": "rgba8",
         "passes": "all", "camera": "above", "lit": False},
        # the 256^3 volume in one 512x512 view, all passes: the small configuration
        {"name": "frame_256cubed", "kind": "frame", "depth": 5, "width": 512, "height": 512, "fmt": "rgba8",
         "passes": "all", "camera": "above", "lit": False},
        # an odd window on half-precision bricks, ray cast only
        {"name": "frame_fp16_odd", "kind": "frame", "depth": 6, "width": 1021, "height": 613, "fmt": "fp16",
         "passes": "raycast", "camera": "above", "lit": False},
        # block-compressed bricks (the memory-saving format), ray cast only
        {"name": "frame_dxt5", "kind": "frame", "depth": 5, "width": 512, "height": 512, "fmt": "dxt5",
         "passes": "raycast", "camera": "above", "lit": False},
        # shaded volume: gradient bricks and Blinn-Phong
        {"name": "frame_lit", "kind": "frame", "depth": 5, "width": 512, "height": 512, "fmt": "rgba8",
         "passes": "all", "camera": "above", "lit": True},
        # a full-HD frame from inside a large terrain, all passes
        {"name": "frame_1080p_low", "kind": "frame", "depth": 9, "width": 1920, "height": 1080, "fmt": "rgba8",
         "passes": "all", "camera": "low", "lit": False},
        # a 4K frame over a large terrain: the largest single draw
        {"name": "frame_2160p", "kind": "frame", "depth": 8, "width": 3840, "height": 2160, "fmt": "rgba8",
         "passes": "all", "camera": "above", "lit": False},
        # the interactive viewer: full-HD flight over a paged terrain, colour read back each frame
        {"name": "flight_paged", "kind": "flight", "depth": 9, "width": 1920, "height": 1080, "fmt": "rgba8",
         "pool_mb": 192},
        # an image server: views of uneven size of terrains of uneven depth in one launch
        {"name": "batch_mixed", "kind": "batch", "depths": "5,6,7,8", "views": 16, "side_min": 128, "side_max": 1024,
         "fmt": "fp16"},
        # a small fit: two small views of a small volume
        {"name": "fit_small", "kind": "fit", "depth": 5, "views": 2, "width": 128, "height": 128,
         "pool_mb": 64},
        # the fit configuration: a 2048^3 volume in 512x512 views
        {"name": "fit_2048cubed", "kind": "fit", "depth": 8, "views": 8, "width": 512, "height": 512,
         "pool_mb": 2048},
        # forward and adjoint of a full-HD frame of a large terrain, sparse gradient rows
        {"name": "adjoint_1080p", "kind": "adjoint", "depth": 9, "width": 1920, "height": 1080, "fmt": "rgba8"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "flight", "batch", "fit", "adjoint"])
    if kind == "frame":
        lit = rng.random() < 0.15
        depth = rng.randint(4, 5) if lit else rng.randint(4, 9)
        return {"kind": "frame", "depth": depth, "width": _log_int(rng, 96, 3840), "height": _log_int(rng, 64, 2160),
                "fmt": rng.choice(["rgba8", "fp32"]) if lit else rng.choice(["rgba8", "rgba8", "fp16", "bf16", "fp32", "dxt5"]),
                "passes": rng.choice(["all", "raycast"]), "camera": rng.choice(["above", "low"]), "lit": lit}
    if kind == "flight":
        return {"kind": "flight", "depth": rng.randint(7, 9), "width": _log_int(rng, 320, 1920),
                "height": _log_int(rng, 200, 1080), "fmt": rng.choice(["rgba8", "rgba8", "fp16"]),
                "pool_mb": rng.randint(96, 256)}
    if kind == "batch":
        deepest = rng.randint(6, 8)
        return {"kind": "batch", "depths": ",".join(str(d) for d in range(deepest - rng.randint(1, 2), deepest + 1)),
                "views": rng.randint(2, 16), "side_min": rng.randint(64, 256), "side_max": rng.randint(257, 1024),
                "fmt": rng.choice(["rgba8", "fp16", "bf16", "fp32"])}
    # even widths: a view's checkpoints are 16-byte records behind 8 bytes a pixel
    if kind == "fit":
        c = {"kind": "fit", "depth": rng.randint(4, 8), "views": rng.randint(1, 8),
             "width": 2 * _log_int(rng, 24, 256), "height": _log_int(rng, 48, 512)}
        # a pool for the bricks of the views, at most those of the volume
        rays = c["views"] * c["width"] * c["height"]
        c["pool_mb"] = min(2048, 16 * 4 ** (c["depth"] - 4), 32 + rays // 1000)
        return c
    return {"kind": "adjoint", "depth": rng.randint(6, 9), "width": 2 * _log_int(rng, 120, 960),
            "height": _log_int(rng, 135, 1080), "fmt": rng.choice(["rgba8", "fp16", "fp32"])}


# ------------------------------------------------------------------ inputs --

class _DeviceBytes:
    """A device range of the context seen by torch."""

    def __init__(self, ptr, nbytes):
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _view(case, octree, heights, seed, frame=0):
    if case.get("camera") == "low":
        return scene.camera_path(seed, heights, 256, case["width"], case["height"])[seed % 256]
    return scene.seeded_view(seed, heights, case["width"], case["height"], frame=frame)


def _renderer(ctx, octree, fmt, pool_bytes):
    """Small volumes preloaded whole, large ones paged on the device."""
    return vv.Renderer(ctx, octree, fmt=fmt, pool_bytes=pool_bytes, preload_all=pool_bytes == 0,
                       alpha_stop=ALPHA_STOP, jitter_seed=JITTER_SEED, device_paging=True)


def _pool_bytes(depth, fmt, deep=1 << 30):
    """0: a pool for every brick; else a pool that holds the bricks of a few views."""
    return 0 if depth <= 6 else int(deep * TEXEL[fmt] / 4)


def prepare(case, seed):
    return {"frame": _prepare_frame, "flight": _prepare_flight, "batch": _prepare_batch, "fit": _prepare_fit,
            "adjoint": _prepare_adjoint}[case["kind"]](case, int(seed))


def _frame_outputs(H, W, passes):
    dev = torch.device("cuda", 0)
    out = {"color": torch.zeros((H, W, 4), dtype=torch.float32, device=dev)}
    if passes == "all":
        out["usage"] = torch.zeros((H, W, 12), dtype=torch.int32, device=dev)
        out["mask"] = torch.zeros((H, W), dtype=torch.int32, device=dev)
        out["requests"] = torch.zeros((H * W, 4), dtype=torch.int32, device=dev)
        out["request_count"] = torch.zeros(1, dtype=torch.int32, device=dev)
    return out


def _prepare_frame(case, seed):
    octree = vv.Octree.terrain(seed=seed, depth=case["depth"], device=0)
    heights = octree.heights()
    cam = _view(case, octree, heights, seed)
    ctx = vv.Context(0)
    st = {"case": case, "ctx": ctx, "octree": octree}
    if case["lit"]:
        words, pool, slots, xyz = scene.resident_scene(octree, case["fmt"])
        ids = np.arange(len(xyz), dtype=np.uint32)
        ctx.upload_nodes(words)
        ctx.create_brickpool(slots, case["fmt"])
        ctx.upload_bricks(ids, pool[:len(xyz)])
        ctx.set_jitter(vv.make_jitter(JITTER_SEED))
        ctx.create_gradpool("fp32")
        st["grads"] = octree.produce_gradients(xyz, "fp32")
        ctx.upload_gradients(ids, st["grads"])
    else:
        st["renderer"] = _renderer(ctx, octree, case["fmt"], _pool_bytes(case["depth"], case["fmt"]))
        if case["depth"] > 6:
            scene.converge_views(st["renderer"], [cam], 32, strict=False)
    st["u"] = vv.compute_uniforms(octree.info, cam, ctx.slots, 1.0, ALPHA_STOP)
    st["u"].compute_lighting = 1 if case["lit"] else 0
    st["out"] = _frame_outputs(case["height"], case["width"], case["passes"])
    return st


def _run_frame(st):
    o = st["out"]
    if st["case"]["passes"] == "all":
        st["ctx"].render(st["u"], color=o["color"].data_ptr(), usage=o["usage"].data_ptr(), mask=o["mask"].data_ptr(),
                         requests=o["requests"].data_ptr(), request_count=o["request_count"].data_ptr(),
                         request_cap=o["requests"].shape[0], passes=vv.VV_PASS_ALL)
    else:
        st["ctx"].render(st["u"], color=o["color"].data_ptr(), passes=vv.VV_PASS_RAYCAST)
    return o


def _prepare_flight(case, seed):
    octree = vv.Octree.terrain(seed=seed, depth=case["depth"], device=0)
    W, H = case["width"], case["height"]
    cams = scene.camera_path(seed, octree.heights(), 256, W, H)[:64:2]
    ctx = vv.Context(0)
    r = _renderer(ctx, octree, case["fmt"], case["pool_mb"] << 20)
    # the pool holds its share of the flight before the first measured frame
    for cam in cams[::4]:
        r.draw(cam)
        r.update()
    host = [torch.zeros((H, W, 4), dtype=torch.float32, pin_memory=True) for _ in range(2)]
    return {"case": case, "ctx": ctx, "octree": octree, "renderer": r, "cams": cams + cams[-2:0:-1], "frame": 0,
            "host": host, "host_np": [h.numpy() for h in host]}


def _run_flight(st):
    r, k = st["renderer"], st["frame"]
    st["frame"] = k + 1
    r.draw(st["cams"][k % len(st["cams"])])
    r.read_color_async(st["host_np"][k & 1])
    r.update()
    s = r.stats()
    return {"color": st["host"][k & 1],
            "service": [int(s[x]) for x in ("requests", "active_pixels", "unique_nodes", "bricks_uploaded",
                                            "resident_bricks", "evictions_total")]}


def _prepare_batch(case, seed):
    rng = np.random.default_rng([case["views"], case["side_max"]])  # the views' sizes are the case's
    dev = torch.device("cuda", 0)
    st = {"case": case, "trees": [], "out": [], "us": [], "tree_of": []}
    items = []
    depths = [int(d) for d in case["depths"].split(",")]
    views = [[] for _ in depths]
    for i in range(case["views"]):
        k = i % len(depths)
        # the first view has the largest side
        w, h = (int(v) for v in rng.integers(case["side_min"], case["side_max"] + 1, size=2))
        views[k].append((i, w if i else case["side_max"], h if i else case["side_max"]))
    slots = {}
    for k, d in enumerate(depths):
        octree = vv.Octree.terrain(seed=seed + k, depth=d, device=0)
        heights = octree.heights()
        ctx = vv.Context(0)
        r = _renderer(ctx, octree, case["fmt"], _pool_bytes(d, case["fmt"], 1 << 29))
        cams = [scene.seeded_view(seed + 100 + i, heights, w, h, frame=i) for i, w, h in views[k]]
        if d > 6 and cams:
            scene.converge_views(r, cams, 16, strict=False)
        st["trees"].append((octree, ctx, r))
        for (i, w, h), cam in zip(views[k], cams):
            slots[i] = (k, cam)
    for i in range(case["views"]):
        k, cam = slots[i]
        octree, ctx, r = st["trees"][k]
        u = vv.compute_uniforms(octree.info, cam, ctx.slots, 1.0, ALPHA_STOP)
        color = torch.zeros((cam.height, cam.width, 4), dtype=torch.float32, device=dev)
        usage = torch.zeros((cam.height, cam.width, 12), dtype=torch.int32, device=dev)
        st["out"].append({"color": color, "usage": usage})
        st["us"].append(u)
        st["tree_of"].append(k)
        items.append((ctx, 0, u, color.data_ptr(), usage.data_ptr()))
    st["batch"] = vv.Batch(st["trees"][0][1], items)
    return st


def _run_batch(st):
    st["batch"].render()
    return st["out"]


def _prepare_fit(case, seed):
    octree = vv.Octree.terrain(seed=seed, depth=case["depth"], device=0)
    heights = octree.heights()
    cams = [scene.seeded_view(seed + v, heights, case["width"], case["height"]) for v in range(case["views"])]
    ctx = vv.Context(0)
    r = _renderer(ctx, octree, "fp32", case["pool_mb"] << 20)
    scene.converge_views(r, cams, 16, strict=False)
    slots = ctx.slots
    us = [vv.compute_uniforms(octree.info, cam, slots, 1.0, ALPHA_STOP) for cam in cams]
    param = diff.pool_tensor_from_context(ctx)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    noisy = param + 0.05 * torch.randn(param.shape, generator=gen, device="cuda")
    with torch.no_grad():
        target = diff.render(noisy, ctx, slots, us)
    torch.cuda.synchronize()
    del noisy
    return {"case": case, "ctx": ctx, "octree": octree, "renderer": r, "us": us, "slots": slots, "target": target,
            "param": param.requires_grad_(True)}


def _run_fit(st):
    image = diff.render(st["param"], st["ctx"], st["slots"], st["us"], PER_RAY)
    loss = ((image - st["target"]) ** 2).mean()
    grad, = torch.autograd.grad(loss, st["param"])
    return {"image": image.detach(), "loss": loss.detach(), "grad": grad}


def _prepare_adjoint(case, seed):
    W, H = case["width"], case["height"]
    dev = torch.device("cuda", 0)
    octree = vv.Octree.terrain(seed=seed, depth=case["depth"], device=0)
    cam = _view(dict(case, camera="low"), octree, octree.heights(), seed)
    ctx = vv.Context(0)
    r = _renderer(ctx, octree, case["fmt"], _pool_bytes(case["depth"], case["fmt"]))
    if case["depth"] > 6:
        scene.converge_views(r, [cam], 32, strict=False)
    u = vv.compute_uniforms(octree.info, cam, ctx.slots, 1.0, ALPHA_STOP)
    n_slots = int(np.prod(ctx.slots))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"case": case, "ctx": ctx, "octree": octree, "renderer": r, "u": u,
          "color": torch.zeros((H, W, 4), dtype=torch.float32, device=dev),
          "target": torch.rand((H, W, 4), generator=gen, device=dev),
          "ckpt": torch.empty(vv.Context.ckpt_bytes(W, H, PER_RAY), dtype=torch.uint8, device=dev),
          "map": torch.full((n_slots,), -1, dtype=torch.int32, device=dev),
          "used": torch.zeros(1, dtype=torch.int32, device=dev)}
    # the rows of the slots that this view touches, in slot order, as a fit
    # that comes back to the view keeps them
    st["n"] = cap = W * H // 10 + 4096
    st["rows"] = torch.zeros((cap, 1000, 4), dtype=torch.float32, device=dev)
    _run_adjoint(st)
    if ctx.device_status():
        raise RuntimeError("the view touches more slots than there are gradient rows")
    hit = torch.nonzero(st["map"] >= 0).flatten()
    st["map"].fill_(-1)
    st["map"][hit] = torch.arange(hit.numel(), dtype=torch.int32, device=dev)
    st["used"].fill_(hit.numel())
    st["n"] = hit.numel()
    st["rows"].zero_()
    torch.cuda.synchronize()
    return st


def _run_adjoint(st):
    ctx, u, color = st["ctx"], st["u"], st["color"]
    ctx.forward_ckpt(u, color.data_ptr(), st["ckpt"].data_ptr(), PER_RAY)
    g = 2.0 * (color - st["target"])
    st["rows"][:st["n"]].zero_()
    ctx.backward_ex(u, g.data_ptr(), st["ckpt"].data_ptr(), PER_RAY, st["rows"].data_ptr(), slot_map=st["map"].data_ptr(),
                    rows_used=st["used"].data_ptr(), rows_cap=st["rows"].shape[0], spread=True)
    return {"color": color, "grad_rows": st["rows"], "slot_map": st["map"]}


def run(state):
    return {"frame": _run_frame, "flight": _run_flight, "batch": _run_batch, "fit": _run_fit,
            "adjoint": _run_adjoint}[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work --

def work(case):
    """What a pass cannot do without, from the sizes alone.  Per pixel: the
    outputs (16 B colour, 48 B usage entries, 4 B mask, about 0.3 requests of
    16 B) and the node words and texels it reads, each once: at one voxel a
    pixel a ray meets about ten texels that no other ray of the frame reads
    first, and about one node word.  A ray composites about 33 samples of 8
    taps and 4 channels (80 operations each) and walks about 26 segments of
    60 operations."""
    kind = case["kind"]
    if kind == "batch":
        mean = ((case["side_min"] + case["side_max"]) / 2.0) ** 2
        rays, out = case["side_max"] ** 2 + (case["views"] - 1) * mean, 64.0
    elif kind == "fit":
        rays, out = case["views"] * case["width"] * case["height"], 16.0
    else:
        rays = case["width"] * case["height"]
        out = 16.0 if case.get("passes") == "raycast" or kind == "adjoint" else 73.0
    texel = TEXEL[case.get("fmt", "fp32")]
    read = 8.0 + 10.0 * texel * (2.0 if case.get("lit") else 1.0)
    flops = 33 * 80.0 + 26 * 60.0
    if kind in ("fit", "adjoint"):
        # the image gradient read, a gradient texel written per texel read,
        # the walk once forward and once backward
        return {"bytes": rays * (out + read + 16.0 + 10.0 * 16.0), "flops": rays * (2.0 * flops + 33 * 80.0)}
    return {"bytes": rays * (out + read), "flops": rays * flops}


# ------------------------------------------------------------ 64-bit values --

def _texels(ctx):
    """The brick pool as (texels, 4) binary64, channels in [0, 1] units."""
    ptr, nbytes = ctx.brickpool_ptr()
    raw = torch.as_tensor(_DeviceBytes(ptr, nbytes), device="cuda")
    fmt = ctx.fmt
    if fmt == vv.VV_FMT_RGBA8:
        return raw.view(-1, 4), 1.0 / 255.0
    if fmt == vv.VV_FMT_FP16:
        return raw.view(torch.float16).view(-1, 4), 1.0
    if fmt == vv.VV_FMT_BF16:
        return raw.view(torch.bfloat16).view(-1, 4), 1.0
    if fmt == vv.VV_FMT_FP32:
        return raw.view(torch.float32).view(-1, 4), 1.0
    return _dxt5_texels(raw), 1.0 / 255.0


def _dxt5_texels(raw):
    """DXT5 slots (90 blocks of 4x4 texels, 3x3 blocks a slice) as RGBA bytes:
    the S3TC interpolation rounded to the nearest, 5 and 6 bit channels
    widened by their high bits."""
    b = raw.view(-1, 16).to(torch.int64)
    word = lambda i, n: sum(b[:, i + k] << (8 * k) for k in range(n))  # noqa: E731
    t = torch.arange(16, device=raw.device)
    a0, a1, ak = b[:, 0:1], b[:, 1:2], (word(2, 6)[:, None] >> (3 * t)) & 7
    wide = torch.where(ak < 2, torch.where(ak == 0, a0, a1), ((8 - ak) * a0 + (ak - 1) * a1 + 3) // 7)
    narrow = torch.where(ak < 2, torch.where(ak == 0, a0, a1), ((6 - ak) * a0 + (ak - 1) * a1 + 2) // 5)
    narrow = torch.where(ak == 6, torch.zeros_like(ak), torch.where(ak == 7, torch.full_like(ak, 255), narrow))
    alpha = torch.where(a0 > a1, wide, narrow)
    c0, c1, ck = word(8, 2)[:, None], word(10, 2)[:, None], (word(12, 4)[:, None] >> (2 * t)) & 3
    out = []
    for shift, bits in ((11, 5), (5, 6), (0, 5)):
        p, q = ((c >> shift) & ((1 << bits) - 1) for c in (c0, c1))
        p, q = ((v << (8 - bits)) | (v >> (2 * bits - 8)) for v in (p, q))
        out.append(torch.where(ck == 0, p, torch.where(ck == 1, q, torch.where(ck == 2, (2 * p + q + 1) // 3,
                                                                               (p + 2 * q + 1) // 3))))
    block = torch.stack(out + [alpha], -1).to(torch.uint8).view(-1, 10, 3, 3, 4, 4, 4)  # slot, z, by, bx, y, x, channel
    return block.permute(0, 1, 2, 4, 3, 5, 6).reshape(-1, 10, 12, 12, 4)[:, :, :10, :10].reshape(-1, 4)


def _lerp32(a, b, t):
    return (t.double() * (b - a).double() + a.double()).float()


def _pow2k(x, k):
    for _ in range(k):
        x = x * x
    return x


class _Cast:
    """One view's ray cast: the sample sequence in binary32, the colour along
    it in binary64 (and in binary32, for the alpha stop)."""

    def __init__(self, ctx, u, texels, scale, words, grads=None, record=False):
        self.dev = torch.device("cuda", 0)
        f = lambda v: torch.tensor(v, dtype=torch.float32, device=self.dev)  # noqa: E731
        self.f, self.u, self.texels, self.scale, self.words = f, u, texels, scale, words
        self.C, self.up, self.left = f(list(u.camera_position)), f(list(u.camera_up)), f(list(u.camera_left))
        self.pdim, self.bdim, self.bstep = f(list(u.brick_pool_dimension)), f(list(u.brick_dimension)), f(list(u.brick_step_vector))
        self.RS, self.rvh, self.lod = f(u.ray_step_size), f(u.root_voxel_half_size), f(u.lod_scalar)
        self.pixel_size, self.astop = f(u.pixel_size), f(u.alpha_stop)
        self.L = u.oct_tree_depth_minus_one
        self.slots = [int(v) // 10 for v in u.brick_pool_dimension]
        self.grads, self.record, self.samples = grads, record, []
        self.jitter = torch.from_numpy(vv.make_jitter(JITTER_SEED)).to(self.dev)

    def dot(self, a, b):
        return a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1] + a[:, 2] * b[:, 2]

    def normalize(self, v):
        return v * (self.f(1.0) / torch.sqrt(self.dot(v, v)))[:, None]

    def origins(self):
        u, f = self.u, self.f
        W, H = u.width, u.height
        px = torch.arange(W, device=self.dev).repeat(H)
        py = torch.arange(H, device=self.dev).repeat_interleave(W)
        fx, fy = (px.float() + 0.5)[:, None], (py.float() + 0.5)[:, None]
        d = (f(list(u.near_origin)) + fx * f(list(u.near_dx))) + fy * f(list(u.near_dy))
        if u.camera_inside:
            return px, py, self.C + d, torch.ones_like(px, dtype=torch.bool)
        lo, hi = f([0.0, 0.0, 0.0]), f([1.0, 1.0, 1.0])
        t0, t1 = (lo - self.C) / d, (hi - self.C) / d
        tn, tf = torch.where(t0 < t1, t0, t1), torch.where(t0 < t1, t1, t0)
        enter = torch.full((px.numel(),), -math.inf, device=self.dev)
        leave = torch.full_like(enter, math.inf)
        axis = torch.full_like(px, -1)
        ok = torch.ones_like(px, dtype=torch.bool)
        for a in range(3):
            moving = d[:, a] != 0
            later = moving & (tn[:, a] > enter)
            enter, axis = torch.where(later, tn[:, a], enter), torch.where(later, torch.full_like(axis, a), axis)
            leave = torch.where(moving & (tf[:, a] < leave), tf[:, a], leave)
            ok &= moving | ((self.C[a] > 0) & (self.C[a] < 1))
        ok &= (axis >= 0) & (enter <= leave) & (enter > 0)
        pos = self.C + d * enter[:, None]
        for a in range(3):
            pos[:, a] = torch.where(axis == a, torch.where(d[:, a] > 0, lo[a], hi[a]), pos[:, a])
        return px, py, pos, ok

    @staticmethod
    def inside(p):
        return ((p > 0) & (p < 1)).all(1)

    def exit_time(self, p, d, lo, hi):
        t = torch.full_like(p[:, 0], 4.0)
        for sign in (-1, 1):
            for a in range(3):
                dn = d[:, a] * sign
                v = (p[:, a] - lo[:, a]) / dn if sign < 0 else -(p[:, a] - hi[:, a]) / dn
                t = torch.where((dn > 0) & (v < t) & (v.abs() > 0), v, t)
        return t

    def descend(self, pos):
        """The node each position's descent stops at."""
        n = pos.shape[0]
        i64 = lambda v: torch.full((n,), v, dtype=torch.int64, device=self.dev)  # noqa: E731
        dz, dy, dx = self.words.shape[:3]
        flat = self.words.view(-1, 2)
        w = flat[0].expand(n, 2)
        rbp, brp, bw = pos.clone(), pos.clone(), w[:, 1].clone()
        depth, bdepth, cell = i64(0), i64(0), torch.zeros((n, 3), dtype=torch.int64, device=self.dev)
        w0, w1 = w[:, 0].clone(), w[:, 1].clone()
        go = torch.arange(n, device=self.dev)  # the positions still descending
        for level in range(self.L + 2):
            c0 = w0[go]
            const, loaded = (c0 & 0x40000000) != 0, (c0 & 0x80000000) != 0
            li = go[loaded]
            bw[li], brp[li], bdepth[li] = w1[li], rbp[li], level
            child = torch.stack([(c0 >> 20) & 1023, (c0 >> 10) & 1023, c0 & 1023], 1)
            down = (const | loaded) & (child != 0).any(1)
            vh = self.rvh * 2.0 ** -level
            uh, lh = self.up * vh, self.left * vh
            p = pos[go]
            ll, ur = self.normalize(p - uh + lh - self.C), self.normalize(p + uh - lh - self.C)
            down &= ~(self.pixel_size > (self.f(1.0) - self.dot(ll, ur)) * self.lod)
            go, child = go[down], child[down]
            if go.numel() == 0:
                break
            b = rbp[go] * 2.0
            o = (b >= 1.0).long()
            rbp[go] = b - o.float()
            cell[go] = 2 * cell[go] + o
            c = child + o
            nw = flat[(c[:, 2] * dy + c[:, 1]) * dx + c[:, 0]]
            w0[go], w1[go] = nw[:, 0], nw[:, 1]
            depth[go] += 1
        return w0, w1, depth, bdepth, bw, brp, cell

    def taps(self, bpos):
        """Texel indices (n, 8) and binary32 weights (n, 3) of a trilinear fetch."""
        t = bpos * self.pdim - 0.5
        t = torch.minimum(torch.maximum(t, self.f(-1.0)), self.pdim)
        fl = torch.floor(t)
        i0 = fl.long()
        ends = []
        for k in (0, 1):
            i = torch.stack([(i0[:, a] + k).clamp(0, self.slots[a] * 10 - 1) for a in range(3)], 1)
            ends.append((i // 10, i % 10))
        idx = []
        for k in range(8):
            s = [ends[(k >> a) & 1][0][:, a] for a in range(3)]
            q = [ends[(k >> a) & 1][1][:, a] for a in range(3)]
            idx.append(((s[2] * self.slots[1] + s[1]) * self.slots[0] + s[0]) * 1000 + (q[2] * 10 + q[1]) * 10 + q[0])
        return torch.stack(idx, 1), t - fl

    def filter(self, texels, scale, idx, w):
        """The fetch in binary32 (as the kernels round it) and in binary64."""
        v = texels[idx.reshape(-1)].view(idx.shape[0], 8, 4)
        out = []
        for x, lerp in ((v.float(), _lerp32), (v.double(), lambda a, b, t: a + t.double() * (b - a))):
            for a in range(3):
                x = lerp(x[:, 0::2], x[:, 1::2], w[:, a, None, None])
            x = x[:, 0]
            out.append(x * self.f(scale) if x.dtype == torch.float32 and scale != 1.0 else x * scale)
        return out

    def light(self, idx, w, d, ldir, src):
        """Blinn-Phong added to binary64 samples from the gradient pool."""
        n = self.filter(self.grads, 1.0, idx, w)[1][:, :3]
        unit = lambda x: x / x.square().sum(1, keepdim=True).sqrt()  # noqa: E731
        n = unit(n)
        ok = ~n.isnan().any(1)
        n = n.nan_to_num()
        half = unit(ldir - d)
        dl = (ldir * n).sum(1).clamp_min(0)
        spec = torch.where(dl > 0, (half * n).sum(1).clamp_min(0) ** 100, torch.zeros_like(dl))
        k = torch.where(ok, 0.05 + dl + spec, torch.zeros_like(dl))
        return torch.cat([src[:, :3] * (1.0 + k)[:, None], src[:, 3:]], 1)

    def composite(self, ray, src32, src64, record=None):
        T32, T64 = 1.0 - self.dst32[ray, 3:], 1.0 - self.dst64[ray, 3:]
        if self.record:
            self.samples.append((ray, T64[:, 0], src64, record))
        self.dst32[ray] = T32 * src32 + self.dst32[ray]
        self.dst64[ray] = T64 * src64 + self.dst64[ray]

    def march(self, ray, n, wstep, step, one_sample):
        """n samples a ray, fewer past the alpha stop; moves self.pos."""
        live = torch.arange(ray.numel(), device=self.dev)
        for i in range(int(n.max()) if n.numel() else 0):
            live = live[n[live] > i]
            if live.numel() == 0:
                break
            r = ray[live]
            self.pos[r] = self.pos[r] + wstep[live]
            full = self.dst32[r, 3] > self.astop
            f, fr = live[full], r[full]
            rem = (n[f] - (i + 1)).float() * step[f]
            self.pos[fr] = self.pos[fr] + self.dir[fr] * rem[:, None]
            live = live[~full]
            one_sample(live, ray[live])

    def run(self):
        px, py, pos, ok = self.origins()
        n, J = px.numel(), self.u.jitter_tex_size
        self.dir = self.normalize(pos - self.C)
        jit = self.jitter[(py % J) * J + px % J].float() / self.f(255.0)
        self.pos = pos + (self.dir * self.RS) * jit[:, None]
        step_b = self.dir * self.bstep
        self.dst32 = torch.zeros((n, 4), dtype=torch.float32, device=self.dev)
        self.dst64 = torch.zeros((n, 4), dtype=torch.float64, device=self.dev)
        active = torch.nonzero(ok & self.inside(self.pos)).flatten()
        while active.numel():
            p = self.pos[active]
            w0, w1, depth, bdepth, bw, brp, cell = self.descend(p)
            s = torch.exp2(-depth.float())[:, None]
            t = self.exit_time(p, self.dir[active], cell.float() * s, (cell + 1).float() * s)
            const, loaded = (w0 & 0x40000000) != 0, (w0 & 0x80000000) != 0
            ratio = torch.exp2((self.L - torch.where(const, depth, bdepth)).float())
            step = self.RS * ratio
            count = (t / step).int() + 1
            # constant nodes: transparent ones are stepped over, the others composited
            byte = (w1 >> 24).float()
            alpha = byte / self.f(255.0)
            skip = const & (alpha < 0.005)
            r = active[skip]
            self.pos[r] = self.pos[r] + self.dir[r] * (count[skip].float() * step[skip])[:, None]
            k = torch.nonzero(const & ~skip).flatten()
            if k.numel():
                rgb = torch.stack([(w1[k] >> sh) & 255 for sh in (0, 8, 16)], 1).float()
                lv = self.L - depth[k]
                a32 = torch.empty_like(alpha[k])
                for v in lv.unique().tolist():
                    a32 = torch.where(lv == v, 1.0 - _pow2k(1.0 - alpha[k], v), a32)
                a64 = 1.0 - (1.0 - byte[k].double() / 255.0) ** torch.exp2(lv.double())
                s32 = torch.cat([rgb / self.f(255.0) * ratio[k, None], a32[:, None]], 1)
                s64 = torch.cat([rgb.double() / 255.0 * ratio[k, None].double(), a64[:, None]], 1)
                self.march(active[k], count[k], self.dir[active[k]] * step[k, None], step[k],
                           lambda j, r: self.composite(r, s32[j], s64[j]))
            # bricks
            k = torch.nonzero(~const).flatten()
            if k.numel():
                r = active[k]
                ptr = torch.stack([(bw[k] >> 20) & 1023, (bw[k] >> 10) & 1023, bw[k] & 1023], 1).float()
                bpos = ptr / self.pdim + (brp[k] * self.bdim) / self.pdim
                ldir = None
                if self.grads is not None:
                    ldir = self.normalize(self.f(list(self.u.light_position)) - self.pos[r]).double()

                def sample(j, r):
                    idx, w = self.taps(bpos[j])
                    s32, s64 = self.filter(self.texels, self.scale, idx, w)
                    s32[:, 3] = 1.0 - (1.0 - s32[:, 3])
                    if ldir is not None:
                        s64 = self.light(idx, w, self.dir[r].double(), ldir[j], s64)
                    self.composite(r, s32, s64, (idx, w) if self.record else None)
                    bpos[j] = bpos[j] + step_b[r]

                self.march(r, count[k], (self.dir[r] * self.RS) * ratio[k, None], step[k], sample)
            done = (self.dst32[active, 3] > self.astop) & (const | loaded)
            active = active[~done & self.inside(self.pos[active])]
        return self.dst64.view(self.u.height, self.u.width, 4)

    def backward(self, g, grad, row_of_texel=None):
        """Adds dL/d(texel) for dL/d(colour) g into grad, (rows, 4) binary64."""
        g = g.reshape(-1, 4).clone()
        for ray, T, src, tap in reversed(self.samples):
            gr = g[ray]
            if tap is not None:
                idx, w = tap
                w = w.double()
                if row_of_texel is not None:
                    idx = row_of_texel(idx)
                d = gr * T[:, None] * self.scale_grad
                for k in range(8):
                    wk = torch.ones_like(T)
                    for a in range(3):
                        wk = wk * (w[:, a] if (k >> a) & 1 else 1.0 - w[:, a])
                    grad.index_add_(0, idx[:, k], d * wk[:, None])
            gr[:, 3] = gr[:, 3] - (gr * src).sum(1)
            g[ray] = gr

    scale_grad = 1.0  # the adjoint's texel gradients are in the units of the filtered value


def _words(ctx):
    return torch.from_numpy(ctx.download_nodes().view(np.int32)).cuda().to(torch.int64) & 0xFFFFFFFF


def exact(case, seed):
    kind = case["kind"]
    # the deep trees' rays cross hundreds of segments: too slow here beyond these sizes
    rays = case.get("width", 0) * case.get("height", 0) * case.get("views", 1)
    if kind == "flight" or (kind != "batch" and case["depth"] > 6 and rays > 3e6) or (kind == "fit" and rays > 1e6):
        return None
    st = prepare(case, seed)
    with torch.no_grad():
        if kind == "frame":
            ctx = st["ctx"]
            grads = torch.from_numpy(st["grads"].view(np.float32).reshape(-1, 4)).cuda() if case["lit"] else None
            texels, scale = _texels(ctx)
            color = _Cast(ctx, st["u"], texels, scale, _words(ctx), grads).run()
            return {"color": color}
        if kind == "batch":
            pools = [_texels(ctx) + (_words(ctx),) for _, ctx, _ in st["trees"]]
            return [{"color": _Cast(None, u, *pools[k]).run()} for u, k in zip(st["us"], st["tree_of"])]
        if kind == "fit":
            texels, words = st["param"].detach().view(-1, 4), _words(st["ctx"])
            grad = torch.zeros(texels.shape, dtype=torch.float64, device=texels.device)
            images, target = [], st["target"].double()
            for v, u in enumerate(st["us"]):
                c = _Cast(None, u, texels, 1.0, words, record=True)
                images.append(c.run())
                c.backward((images[v] - target[v]) * (2.0 / target.numel()), grad)
            image = torch.stack(images)
            return {"image": image, "loss": (image - target).square().mean(), "grad": grad.view(st["param"].shape)}
        ctx = st["ctx"]
        texels, scale = _texels(ctx)
        c = _Cast(None, st["u"], texels, scale, _words(ctx), record=True)
        color = c.run()
        rows = torch.zeros((st["rows"].shape[0] * 1000, 4), dtype=torch.float64, device=color.device)
        slot_row = st["map"].long()
        c.backward(2.0 * (color - st["target"].double()), rows, lambda i: slot_row[i // 1000] * 1000 + i % 1000)
        return {"color": color, "grad_rows": rows.view(st["rows"].shape), "slot_map": None}
