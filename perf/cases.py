"""Workloads of the volume raycaster, for measuring it from outside.

Each case is one kind of call that programs built on this framework make:

  frame      a frame of an animation loop: device entry/exit images (or an
             analytic proxy box) in, a device image out
  still      the blocking call of the README: analytic proxy box, host image
  tf_edit    a frame after the user moved a transfer-function key: bake, new
             table on the device, frame
  time_step  the next time step of a series: voxels in host memory are
             uploaded and their first frame is shown
  batch      many mixed requests in one captured launch
  upsample   the upsampler network on a half-resolution frame
  conv       one convolution layer in training: forward, data gradient,
             weight gradient

Volumes are made on the GPU from the seed: Gaussian blobs, CT-like nested
ellipsoid shells with noise, sparse tubes. Cameras orbit the volume.
"""
import ctypes
import math
import os
import random

import numpy as np
import torch

import voreen_gb300 as v
from voreen_gb300 import learned

SCALE = {"u8": 255, "u16": 4095, "f32": 1}          # stored value of unit intensity
RANGE = {"u8": 255.0, "u16": 65535.0, "f32": 1.0}   # what the march normalises by
BYTES = {"u8": 1, "u16": 2, "f32": 4}
COMPOSITING = {"dvr": v.DVR, "mip": v.MIP, "iso": v.ISO, "mop": v.MOP, "mida": v.MIDA, "fhp": v.FHP, "fhn": v.FHN}
SHELLS = (200, 1000, 1800, 2600, 3200, 4000)
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(learned.__file__)), "weights", "upsampler_ct.npz")


def _frame(name, content, dims, dtype, image, **more):
    c = {"kind": "frame", "content": content, "x": dims[0], "y": dims[1], "z": dims[2], "dtype": dtype,
         "width": image[0], "height": image[1], "rate": 2.0, "compositing": "dvr", "phong": False, "tf_width": 4096,
         "out": "rgba8", "buffers": False, "preint": False, "distance": 1.25}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a thumbnail of a small volume: launches and the latency of one short ray march
        _frame("thumbnail_64_u8", "blobs", (64, 64, 64), "u8", (256, 256), tf_width=256, distance=1.6),
        # the README's first call on the plain DVR configuration (128^3 u8 blobs, 512x512)
        _frame("still_128_u8", "blobs", (128, 128, 128), "u8", (512, 512), kind="still", tf_width=256, out="rgba32f",
               distance=2.5),
        # the headline configuration: CT-like 512^3 u16, Phong DVR, 1080p, entry/exit images on the device
        _frame("ct_512_u16_phong", "shells", (512, 512, 512), "u16", (1920, 1080), phong=True, buffers=True),
        # the same volume under maximum intensity projection (no early ray termination)
        _frame("ct_512_u16_mip", "shells", (512, 512, 512), "u16", (1920, 1080), compositing="mip", buffers=True),
        # the same volume with a pre-integrated transfer function
        _frame("ct_512_u16_preint", "shells", (512, 512, 512), "u16", (1920, 1080), phong=True, preint=True),
        # float voxels, odd sizes on every side, shaded isosurface, float image
        _frame("iso_odd_f32", "blobs", (253, 187, 201), "f32", (1023, 769), compositing="iso", phong=True,
               out="rgba32f", tf_width=1024),
        # dragging a transfer-function key: each frame has a table that the library has not seen
        _frame("tf_edit_512_u16", "shells", (512, 512, 512), "u16", (1920, 1080), kind="tf_edit", phong=True),
        # playing a time series from host memory: upload and first frame of each step
        _frame("time_step_512_u16", "shells", (512, 512, 512), "u16", (1024, 1024), kind="time_step", phong=True),
        # the largest: 8 GiB of sparse tubes at 4K
        _frame("tubes_2048_u16_4k", "tubes", (2048, 2048, 1024), "u16", (3840, 2160), phong=True, rate=1.5,
               distance=1.2),
        # a render service's queue: 64 requests of mixed sizes and types in one launch
        {"name": "batch_64", "kind": "batch", "requests": 64, "largest": 512},
        # the upsampler on the half-resolution frame of a 1080p view
        {"name": "upsample_1080p", "kind": "upsample", "height": 540, "width": 960},
        # training of one of the upsampler's layers on 8 crops
        {"name": "conv_64_64_train", "kind": "conv", "n": 8, "height": 96, "width": 96, "cin": 64, "cout": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "frame", "still", "tf_edit", "time_step", "batch", "upsample", "conv"))
    if kind == "batch":
        return {"kind": kind, "requests": rng.randint(3, 48), "largest": rng.choice((256, 384, 512))}
    if kind == "upsample":
        return {"kind": kind, "height": 4 * _log(rng, 20, 250), "width": 4 * _log(rng, 20, 450)}
    if kind == "conv":
        return {"kind": kind, "n": rng.randint(1, 16), "height": _log(rng, 24, 160), "width": _log(rng, 24, 160),
                "cin": rng.choice((16, 32, 64, 128)), "cout": rng.choice((16, 32, 64, 128))}
    content = rng.choice(("blobs", "shells", "shells", "tubes"))
    dtype = "u16" if content == "tubes" else rng.choice(("u8", "u16", "u16", "f32"))
    edge = _log(rng, 40, 400 if kind == "time_step" else 640)
    dims = [max(24, int(edge * rng.uniform(0.6, 1.0))) for _ in range(3)]
    width = _log(rng, 120, 2000)
    image = (width, max(64, int(width * rng.uniform(0.5, 1.0))))
    compositing, phong, preint = "dvr", rng.random() < 0.6, False
    if kind == "frame" and rng.random() < 0.5:
        compositing = rng.choice(("mip", "mip", "iso", "mop", "mida", "fhp", "fhn"))
        phong = phong and compositing in ("iso", "mida")
    elif kind == "frame":
        preint = rng.random() < 0.25
    return _frame(None, content, dims, dtype, image, kind=kind, rate=rng.choice((1.0, 1.5, 2.0, 2.0, 3.0)),
                  compositing=compositing, phong=phong, tf_width=256 if dtype == "u8" else rng.choice((1024, 4096)),
                  out=rng.choice(("rgba8", "rgba8", "rgba32f")), buffers=kind == "frame" and rng.random() < 0.4,
                  preint=preint, distance=round(rng.uniform(1.1, 2.2), 2))


# ---- inputs ----------------------------------------------------------------------


def _blobs(dims, rng, gen):
    """Sum of 8 isotropic Gaussians plus uniform noise, in unit intensity."""
    X, Y, Z = dims
    out = torch.zeros((Z, Y, X), device="cuda")
    for _ in range(8):
        c = [rng.uniform(0.2, 0.8) * d for d in dims]
        k = -0.5 / rng.uniform(4.0, 16.0) ** 2
        ex, ey, ez = (torch.exp(k * (torch.arange(d, device="cuda") - p) ** 2) for d, p in zip(dims, c))
        out += rng.uniform(80.0, 255.0) / 255.0 * ez[:, None, None] * ey[None, :, None] * ex
    out += 10.0 / 255.0 * torch.rand(out.shape, generator=gen, device="cuda")
    return out.clamp_(max=1.0)


def _shells(dims, rng, gen):
    """Six nested, rotated ellipsoid shells on background 0 plus Gaussian noise, in unit intensity."""
    c = [d * (0.5 + rng.uniform(-0.05, 0.05)) for d in dims]
    a = [d * rng.uniform(0.30, 0.45) for d in dims]
    q, _ = np.linalg.qr(np.array([[rng.gauss(0, 1) for _ in range(3)] for _ in range(3)]))
    unit = min(1.0, max(min(dims) / 512.0, 0.25))
    px, py, pz = (torch.arange(d, device="cuda", dtype=torch.float32) - o for d, o in zip(dims, c))
    axes = [float(r[2]) * pz[:, None, None] + float(r[1]) * py[None, :, None] + float(r[0]) * px for r in q]
    axes = [x * x for x in axes]
    out = torch.zeros((dims[2], dims[1], dims[0]), device="cuda")
    for k, value in enumerate(SHELLS):  # the inner shells lie inside and are written last
        th = rng.uniform(3.0, 12.0) * unit
        outer = [x * (1.0 - 0.14 * k) for x in a]
        for radii, val in ((outer, value / 4095.0), ([max(x - th, 0.5) for x in outer], 0.0)):
            r2 = axes[0] / radii[0] ** 2
            for j in (1, 2):
                r2 += axes[j] / radii[j] ** 2
            out.masked_fill_(r2 <= 1.0, val)
    del axes, r2
    out += 20.0 / 4095.0 * torch.randn(out.shape, generator=gen, device="cuda")
    return out.clamp_(0.0, 1.0)


def _voxels(content, dims, dtype, seed):
    """(Z, Y, X) CUDA tensor of stored values, and its smallest and largest value."""
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if content == "tubes":
        n = max(8, round(500 * dims[0] * dims[1] * dims[2] / 2.0 ** 32))
        vox = v.synth_tubes_device(dims, n, seed)
        torch.cuda.synchronize()
        return vox, 0, 4095
    unit = (_blobs if content == "blobs" else _shells)(dims, rng, gen)
    if dtype == "f32":
        return unit, float(unit.min()), float(unit.max())
    unit.mul_(SCALE[dtype]).round_()
    mn, mx = int(unit.min()), int(unit.max())
    if dtype == "u8":
        return unit.to(torch.uint8), mn, mx
    return unit.to(torch.int16).view(torch.uint16), mn, mx


def _trapezoids(rng, centres, alpha, top, ramp):
    """Keys (position, RGBA8): one trapezoid of opacity at each centre."""
    keys = []
    for c in sorted(centres):
        t, r, a = rng.uniform(*top), rng.uniform(*ramp), round(255 * rng.uniform(*alpha))
        col = tuple(rng.randint(60, 255) for _ in range(3))
        for p, o in ((c - t - r, 0), (c - t, a), (c + t, a), (c + t + r, 0)):
            p = min(1.0, max(0.0, p))
            keys.append((p if not keys or p > keys[-1][0] else min(1.0, keys[-1][0] + 1e-6), (*col, o)))
    return keys


def _tf_keys(content, dtype, mn, mx, seed):
    """The transfer function that goes with a volume, over the domain [mn, mx] of its stored values."""
    rng = random.Random(seed + 7)
    lo, hi = mn / SCALE[dtype], mx / SCALE[dtype]
    at = lambda x: (x - lo) / (hi - lo)  # noqa: E731
    if content == "blobs":  # opacity 0 below intensity 40 of 255, then a ramp; blue to red
        t = at(40.0 / 255.0 + rng.uniform(0.0, 0.04))
        col = lambda a: (round(255 * a), 0, round(255 * (1 - a)))  # noqa: E731
        return [(0.0, (*col(0.0), 0)), (t, (*col(t), 0)), (1.0, (*col(1.0), 153))]
    if content == "shells":
        peaks = [at(p / 4095.0) for p in rng.sample(SHELLS, 5)]
        return _trapezoids(rng, peaks, (0.1, 0.8), (0.004, 0.015), (0.006, 0.02))
    peaks = [at(rng.uniform(1600 + 1200 * k, 2600 + 1200 * k) / 4095.0) for k in range(2)]
    return _trapezoids(rng, peaks, (0.2, 0.7), (0.01, 0.03), (0.02, 0.05))


def _table(keys, width):
    """The keys as an RGBA8 table, interpolated linearly."""
    x = np.linspace(0.0, 1.0, width)
    p = [k[0] for k in keys]
    return np.stack([np.interp(x, p, [k[1][c] for k in keys]) for c in range(4)], 1).astype(np.uint8)


def _spacing(content):
    return (0.7, 0.7, 1.0) if content == "shells" else (1.0, 1.0, 1.0)


def _orbit(dims, spacing, azimuth, elevation, distance):
    """Camera position, focus, near and far: `distance` box diagonals from the box's centre."""
    c = [0.5 * (d - 1) * s for d, s in zip(dims, spacing)]
    diag = math.sqrt(sum((d * s) ** 2 for d, s in zip(dims, spacing)))
    az, el, r = math.radians(azimuth), math.radians(elevation), distance * diag
    pos = (c[0] + r * math.sin(az) * math.cos(el), c[1] + r * math.sin(el), c[2] + r * math.cos(az) * math.cos(el))
    return pos, tuple(c), max(1e-3, r - diag), r + diag


def _view(case, seed):
    rng = random.Random(seed + 3)
    return _orbit((case["x"], case["y"], case["z"]), _spacing(case["content"]), 35.0 + rng.uniform(-10, 10),
                  25.0 + rng.uniform(-5, 5), case["distance"])


def _params(case, view):
    pos, focus, near, far = view
    p = v.default_params(case["width"], case["height"])
    p.sampling_rate = case["rate"]
    p.compositing = COMPOSITING[case["compositing"]]
    p.shading = v.SHADE_PHONG if case["phong"] else v.SHADE_NONE
    p.camera = v.make_camera(pos, focus, near=near, far=far)
    p.light_position[:] = [*pos, 1.0]
    p.entry_exit_mode = v.EE_BUFFERS if case["buffers"] else v.EE_ANALYTIC
    p.iso_value = 0.4
    p.mida_gamma = 0.3
    return p


class _Program:
    """A user's program: its context, and torch's stream ordered around the context's."""

    def __init__(self):
        self.ctx = v.Context(0)
        self.stream = torch.cuda.ExternalStream(self.ctx.stream)

    def __enter__(self):
        self.stream.wait_stream(torch.cuda.current_stream())

    def __exit__(self, *a):
        torch.cuda.current_stream().wait_stream(self.stream)


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    if case["kind"] == "upsample":
        return _prepare_upsample(case, seed)
    if case["kind"] == "conv":
        return _prepare_conv(case, seed)
    dims, content = (case["x"], case["y"], case["z"]), case["content"]
    spacing = _spacing(content)
    vox, mn, mx = _voxels(content, dims, case["dtype"], seed)
    torch.cuda.synchronize()
    prog = _Program()
    s = {"kind": case["kind"], "program": prog, "params": _params(case, _view(case, seed)), "width": case["tf_width"],
         "keys": _tf_keys(content, case["dtype"], mn, mx, seed), "spacing": spacing,
         "format": v.OUT_RGBA8 if case["out"] == "rgba8" else v.OUT_RGBA32F, "entry": None, "exit": None}
    s["domain"] = tuple(float(np.float32(x) / np.float32(RANGE[case["dtype"]])) for x in (mn, mx))
    shape = (case["height"], case["width"], 4)
    if case["kind"] != "still":
        s["out"] = torch.empty(shape, dtype=torch.uint8 if case["out"] == "rgba8" else torch.float32, device="cuda")
    if case["kind"] == "time_step":
        s["voxels"] = vox.cpu().numpy()
        s["tf"] = v.TransferFunction(prog.ctx, _table(s["keys"], s["width"]), s["domain"])
        return s
    s["volume"] = v.Volume(prog.ctx, vox, spacing)
    if case["kind"] == "tf_edit":
        return s
    s["tf"] = v.TransferFunction(prog.ctx, _table(s["keys"], s["width"]), s["domain"])
    if case["preint"]:
        res = v.PreIntegrationTable.resolution(s["width"])
        s["preint"] = v.PreIntegrationTable(prog.ctx, _table(s["keys"], res),
                                            v.sampling_step(s["volume"], case["rate"]))
        s["tf"].set_preintegration(s["preint"])
        s["params"].classification = v.CLASSIFY_PREINTEGRATED
    if case["buffers"]:
        e, x = v.entry_exit(prog.ctx, s["volume"], s["params"])
        s["entry"], s["exit"] = torch.from_numpy(e).cuda(), torch.from_numpy(x).cuda()
    return s


def _prepare_batch(case, seed):
    """Requests as a render service gets them: volumes of mixed sizes, types and contents shared by several
    requests, their own cameras, transfer functions and image sizes; all images in one slab."""
    rng = random.Random(seed)
    prog = _Program()
    plan, volumes, items = _batch_plan(case, rng), {}, []
    slab = torch.empty(sum(r["width"] * r["height"] for r in plan) * 4, dtype=torch.uint8, device="cuda")
    at = 0
    for r in plan:
        key = (r["dims"], r["dtype"], r["content"])
        if key not in volumes:
            vox, _, _ = _voxels(r["content"], r["dims"], r["dtype"], seed * 100 + len(volumes))
            torch.cuda.synchronize()
            volumes[key] = v.Volume(prog.ctx, vox, (1.0, 1.0, 1.0))
            del vox
        vol = volumes[key]
        slots = sorted(rng.sample(range(9), 3))
        centres = [0.15 + 0.8 * (k + rng.uniform(0.3, 0.7)) / 9 for k in slots]
        keys = _trapezoids(rng, centres, (0.15, 0.7), (0.01, 0.03), (0.01, 0.03))
        tf = v.TransferFunction(prog.ctx, _table(keys, r["tf_width"]), vol.minmax())
        pos, focus, near, far = _orbit(r["dims"], (1.0, 1.0, 1.0), rng.uniform(0, 360), rng.uniform(-60, 60),
                                       rng.uniform(1.1, 2.0))
        p = v.default_params(r["width"], r["height"])
        p.shading, p.entry_exit_mode = v.SHADE_PHONG, v.EE_ANALYTIC
        p.camera = v.make_camera(pos, focus, near=near, far=far)
        p.light_position[:] = [*pos, 1.0]
        n = r["width"] * r["height"] * 4
        items.append((vol, tf, p, slab[at:at + n], v.OUT_RGBA8))
        at += n
    torch.cuda.synchronize()
    return {"kind": "batch", "program": prog, "batch": v.Batch(prog.ctx, items), "slab": slab}


def _batch_plan(case, rng):
    dims = [d for d in ((64, 64, 64), (128, 128, 128), (256, 256, 256), (384, 256, 200), (512, 512, 512))
            if max(d) <= case["largest"]]
    images = ((256, 256), (512, 512), (1024, 1024), (1920, 1080), (2048, 2048))
    plan = []
    for i in range(case["requests"]):
        w, h = images[i % len(images)]
        plan.append({"dims": dims[i % len(dims)], "dtype": rng.choice(("u8", "u16", "f32")),
                     "content": rng.choice(("blobs", "shells")), "width": w, "height": h,
                     "tf_width": rng.choice((256, 4096))})
    order = list(range(len(plan)))  # every size against every image size
    rng.shuffle(order)
    return [dict(plan[i], dims=plan[j]["dims"]) for i, j in enumerate(order)]


def _upsample_inputs(case, seed):
    """A half-resolution march as the network sees it: colour and opacity of smooth objects with edges on an
    empty background, first-hit depth and gradient."""
    h, w = case["height"], case["width"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    yy = torch.linspace(-1, 1, h, device="cuda")[:, None]
    xx = torch.linspace(-1, 1, w, device="cuda")[None, :]
    r = torch.sqrt(xx * xx + yy * yy) + 0.1 * torch.sin(5 * xx + 3 * yy)
    low = torch.rand((1, 5, 12, 20), generator=gen, device="cuda")
    tex = torch.nn.functional.interpolate(low, (h, w), mode="bilinear", align_corners=False)[0]
    alpha = ((r < 0.9).float() * (0.4 + 0.5 * tex[3]) * (1.0 - 0.6 * ((r > 0.5) & (r < 0.55)).float()))[..., None]
    rgba = torch.cat([tex[:3].permute(1, 2, 0) * alpha, alpha], -1)[None].contiguous()
    depth = torch.where(alpha > 0, 0.2 + 0.4 * r[..., None], torch.ones_like(alpha))
    x0 = torch.zeros((1, h, w, 16), device="cuda")
    x0[..., :4] = rgba
    x0[..., 4:5] = depth
    x0[..., 5:6] = alpha * tex[4][..., None]
    return x0.to(torch.bfloat16), rgba


def _prepare_upsample(case, seed):
    x0, base = _upsample_inputs(case, seed)
    net = learned.UNet(seed=0)
    net.load(WEIGHTS)
    return {"kind": "upsample", "net": net, "x0": x0, "base": base,
            "out": torch.empty((1, 2 * case["height"], 2 * case["width"], 4), device="cuda")}


def _conv_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w, ci, co = (case[k] for k in ("n", "height", "width", "cin", "cout"))
    rand = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    x = rand(n, h, w, ci)
    x = torch.where(x > 0, x, 0.05 * x).to(torch.bfloat16)  # what a leaky ReLU leaves
    dy = (rand(n, h, w, co) * 1e-2).to(torch.bfloat16)
    wt = (rand(co, 3, 3, ci) * math.sqrt(2.0 / (9 * ci))).to(torch.bfloat16)
    return x, dy, wt, rand(co) * 0.1


def _prepare_conv(case, seed):
    x, dy, wt, bias = _conv_inputs(case, seed)
    flipped = torch.empty((case["cin"], 3, 3, case["cout"]), dtype=torch.bfloat16, device="cuda")
    if v.lib().vrc_nn_flip_weights(_at(wt), case["cout"], case["cin"], _at(flipped), _current()) != 0:
        raise RuntimeError("vrc_nn_flip_weights failed")
    s = {"kind": "conv", "x": x, "dy": dy, "w": wt, "flipped": flipped, "bias": bias, "y": torch.empty_like(dy),
         "dx": torch.empty_like(x), "dw": torch.empty(wt.shape, device="cuda"), "db": torch.empty_like(bias)}
    s.update({k: case[k] for k in ("n", "height", "width", "cin", "cout")})
    return s


def _at(t):
    return ctypes.c_void_p(t.data_ptr())


def _current():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# ---- one pass ---------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "conv":
        return _run_conv(s)
    if kind == "upsample":
        return s["net"].infer_tc(s["x0"], s["base"], s["out"])
    prog = s["program"]
    if kind == "batch":
        with prog:
            s["batch"].launch()
        return s["slab"]
    if kind == "still":
        image, _ = v.render(prog.ctx, s["volume"], s["tf"], s["params"], out_format=s["format"])
        return image
    if kind == "time_step":
        volume = v.Volume(prog.ctx, s["voxels"], s["spacing"])
        with prog:
            v.render_async(prog.ctx, volume, s["tf"], s["params"], None, None, s["out"], s["format"])
        lo, hi = volume.minmax()
        volume.close()
        return {"image": s["out"], "min": lo, "max": hi}
    if kind == "tf_edit":
        table = v.TransferFunction.bake(s["keys"], s["width"])
        tf = v.TransferFunction(prog.ctx, table, s["domain"])
        with prog:
            v.render_async(prog.ctx, s["volume"], tf, s["params"], None, None, s["out"], s["format"])
        tf.close()
        return s["out"]
    with prog:
        v.render_async(prog.ctx, s["volume"], s["tf"], s["params"], s["entry"], s["exit"], s["out"], s["format"])
    return s["out"]


def _run_conv(s):
    L, n, h, w, ci, co = v.lib(), s["n"], s["height"], s["width"], s["cin"], s["cout"]
    st = _current()
    s["dw"].zero_()
    s["db"].zero_()
    ok = L.vrc_nn_conv3x3_fwd(_at(s["x"]), n, h, w, ci, _at(s["w"]), _at(s["bias"]), co, 2, _at(s["y"]), 0, st)
    ok |= L.vrc_nn_conv3x3_fwd(_at(s["dy"]), n, h, w, co, _at(s["flipped"]), None, ci, 0, _at(s["dx"]), 0, st)
    ok |= L.vrc_nn_conv3x3_wgrad(_at(s["x"]), _at(s["dy"]), n, h, w, ci, co, _at(s["dw"]), _at(s["db"]), st)
    if ok:
        raise RuntimeError("a convolution kernel failed")
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def work(case):
    kind = case["kind"]
    if kind == "conv":
        n, h, w, ci, co = (case[k] for k in ("n", "height", "width", "cin", "cout"))
        return {"bytes": 2.0 * n * h * w * 2 * (ci + co) + 9 * ci * co * (2 + 2 + 4) + 8 * co,
                "flops": 3 * 18.0 * n * h * w * ci * co}
    if kind == "upsample":
        px = case["height"] * case["width"]
        macs = sum(9 * ci * co / {"enc2": 4, "dec2": 4, "bota": 16, "botb": 16}.get(name[:4], 1)
                   for name, ci, co, _ in learned.LAYERS)
        weights = sum(9 * ci * co * 2 + 4 * co for _, ci, co, _ in learned.LAYERS)
        return {"bytes": px * (16 * 2 + 16 + 64.0) + weights, "flops": 2.0 * px * macs}
    if kind == "batch":
        plan = _batch_plan(case, random.Random(0))
        volumes = {(r["dims"], r["dtype"], r["content"]): r["dims"][0] * r["dims"][1] * r["dims"][2] * BYTES[r["dtype"]]
                   for r in plan}
        return {"bytes": float(sum(volumes.values()) + sum(4 * r["width"] * r["height"] for r in plan)), "flops": 0.0}
    px = case["width"] * case["height"]
    per_px = (4 if case["out"] == "rgba8" else 16) + (32 if case["buffers"] else 0)
    return {"bytes": float(case["x"] * case["y"] * case["z"] * BYTES[case["dtype"]] + px * per_px), "flops": 0.0}


# ---- what run returns, in 64 bits ---------------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        return _exact_conv(case, seed)
    if kind == "upsample":
        return _exact_upsample(case, seed)
    if kind == "batch":
        return None
    if kind == "time_step":
        _, mn, mx = _voxels(case["content"], (case["x"], case["y"], case["z"]), case["dtype"], seed)
        if case["content"] == "tubes":
            return None
        image = _exact_frame(case, seed) if case["out"] == "rgba32f" else None
        return {"image": image, "min": mn / RANGE[case["dtype"]], "max": mx / RANGE[case["dtype"]]}
    if case["out"] != "rgba32f" or kind == "tf_edit" or case["preint"]:
        return None
    return _exact_frame(case, seed)


def _exact_frame(case, seed):
    """The frame by a plain march in float64: nearest transfer-function entry, trilinear samples, central
    differences, Phong with the light at the camera, front-to-back compositing with early termination at 0.95."""
    W, H, dims = case["width"], case["height"], (case["x"], case["y"], case["z"])
    comp, step = case["compositing"], 1.0 / (max(case["x"], case["y"], case["z"]) * case["rate"])
    if comp not in ("dvr", "mip", "iso") or case["content"] == "tubes":
        return None
    if W * H / step * (6.0 if case["phong"] else 1.0) > 6e9:
        return None
    f64 = dict(dtype=torch.float64, device="cuda")
    vox, mn, mx = _voxels(case["content"], dims, case["dtype"], seed)
    flat = (vox.view(torch.int16) if case["dtype"] == "u16" else vox).reshape(-1).to(torch.float64)
    flat = flat / RANGE[case["dtype"]]
    del vox
    lo, hi = (float(np.float32(x) / np.float32(RANGE[case["dtype"]])) for x in (mn, mx))
    table = torch.from_numpy(_table(_tf_keys(case["content"], case["dtype"], mn, mx, seed), case["tf_width"])).to(**f64) / 255.0
    spacing = torch.tensor(np.float32(_spacing(case["content"])).astype(np.float64), **f64)
    dim = torch.tensor([float(d) for d in dims], **f64)
    pos, focus, near, far = _view(case, seed)
    pos, focus = (np.float32(p).astype(np.float64) for p in (pos, focus))
    near, far = float(np.float32(near)), float(np.float32(far))
    # rays through the pixel centres, in texture coordinates
    look = (focus - pos) / np.linalg.norm(focus - pos)
    right = np.cross(look, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, look)
    ty = math.tan(math.radians(22.5))
    if W < H:
        ty = ty * H / W
    tx = ty * W / H
    to = lambda a: torch.tensor(a, **f64)  # noqa: E731
    nx = ((torch.arange(W, **f64) + 0.5) / W * 2 - 1) * tx
    ny = ((torch.arange(H, **f64) + 0.5) / H * 2 - 1) * ty
    ray = (to(look) + nx[None, :, None] * to(right) + ny[:, None, None] * to(up)).reshape(-1, 3)
    size = spacing * dim
    org = (to(pos) + 0.5 * spacing) / size
    o, d = org + near * ray / size, (far - near) * ray / size
    a, b = (0.0 - o) / d, (1.0 - o) / d
    s0 = torch.minimum(a, b).amax(1).clamp(min=0.0)
    s1 = torch.maximum(a, b).amin(1).clamp(max=1.0)
    hit = s0 < s1
    zero = torch.zeros((), **f64)
    entry = torch.where(hit[:, None], (o + s0[:, None] * d).clamp(0, 1), zero)
    leave = torch.where(hit[:, None], (o + s1[:, None] * d).clamp(0, 1), zero)
    end = (leave - entry).norm(dim=1)
    dirs = (leave - entry) / end.clamp(min=1e-300)[:, None]

    def at(p):  # trilinear value at voxel positions
        i = p.floor()
        f = p - i
        i = i.long()
        j = torch.minimum(i + 1, (dim - 1).long())
        r = 0.0
        for k in range(8):
            pick = [j if k >> ax & 1 else i for ax in range(3)]
            w = 1.0
            for ax in range(3):
                w = w * (f[:, ax] if k >> ax & 1 else 1.0 - f[:, ax])
            r = r + w * flat[(pick[2][:, 2] * dims[1] + pick[1][:, 1]) * dims[0] + pick[0][:, 0]]
        return r

    def voxel(s):
        return torch.minimum((s * dim - 0.5).clamp(min=0.0), dim - 1)

    def unit(x):
        n = x.norm(dim=1, keepdim=True)
        return torch.where(n > 0, x / n.clamp(min=1e-300), zero)

    def shade(rays, s, t, col):
        g = torch.empty_like(s)
        for ax in range(3):
            e = torch.zeros(3, **f64)
            e[ax] = 1.0 / dims[ax]
            g[:, ax] = (at(voxel(s - e)) - at(voxel(s + e))) * 0.5 / spacing[ax]
        if t == 0.0:  # on the proxy's face: the normal of the face, from the neighbours' entry points
            x, y = rays % W, rays // W
            v0 = unit(entry[y * W + (x + 2).clamp(max=W - 1)] - s)
            v1 = unit(entry[(y + 2).clamp(max=H - 1) * W + x] - s)
            g = torch.linalg.cross(v0, v1)
            g = torch.where((g * dirs[rays]).sum(1, keepdim=True) < 0, g, -g)
        world = (s * dim - 0.5) * spacing
        n, light = unit(g), unit(to(pos) - world)
        ndl = (n * light).sum(1, keepdim=True).clamp(min=0)
        ndh = (n * unit(light + light)).sum(1, keepdim=True).clamp(min=0)
        return 0.4 * col + 0.8 * col * ndl + 0.6 * ndh ** 60.0

    out = torch.zeros((W * H, 4), **f64)
    rays = torch.nonzero(hit).reshape(-1)
    res = torch.zeros((len(rays), 4), **f64)
    best = torch.zeros(len(rays), **f64)
    alphas = 1.0 - (1.0 - table[:, 3]) ** (step * 200.0) if comp == "dvr" else table[:, 3]
    t = 0.0
    while len(rays):
        s = entry[rays] + t * dirs[rays]
        value = at(voxel(s))
        x = ((value - lo) / (hi - lo)).clamp(0, 1)
        k = (x * (case["tf_width"] - 1) + 0.5).floor().long()
        alpha = alphas[k]
        col = table[k][:, :3]
        vis = torch.nonzero(alpha > 0).reshape(-1)
        if comp == "iso":
            vis = vis[(alpha[vis] - 0.4).abs() <= 0.02]
        elif comp == "mip":
            vis = vis[value[vis] > best[vis]]
            best[vis] = value[vis]
        col, alpha = col[vis], alpha[vis][:, None]
        if case["phong"] and len(vis):
            col = shade(rays[vis], s[vis], t, col)
        if comp == "dvr":
            w = (1.0 - res[vis, 3:]) * alpha
            res[vis] = res[vis] + torch.cat([w * col, w], 1)
        else:
            res[vis] = torch.cat([col, torch.ones_like(alpha) if comp == "iso" else alpha], 1)
        t += step
        done = end[rays] < t
        if comp != "mip":
            opaque = res[:, 3] >= 0.95
            res[opaque, 3] = 1.0
            done = done | opaque
        out[rays[done]] = res[done]
        live = ~done
        rays, res, best = rays[live], res[live], best[live]
    out = out.reshape(H, W, 4)
    return out.cpu().numpy() if case["kind"] == "still" else out


def _conv64(x, w):
    """3x3 convolution with zero borders, NHWC, weights [Cout][3][3][Cin]."""
    n, h, wd, ci = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = 0.0
    for ky in range(3):
        for kx in range(3):
            y = y + p[:, ky:ky + h, kx:kx + wd].reshape(-1, ci) @ w[:, ky, kx].T
    return y.reshape(n, h, wd, w.shape[0])


def _leaky(x):
    return torch.where(x > 0, x, float(np.float32(0.05)) * x)


def _exact_conv(case, seed):
    x, dy, w, b = (t.to(torch.float64) for t in _conv_inputs(case, seed))
    n, h, wd = case["n"], case["height"], case["width"]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    g = dy.reshape(-1, case["cout"])
    dw = torch.stack([torch.stack([g.T @ p[:, ky:ky + h, kx:kx + wd].reshape(-1, case["cin"]) for kx in range(3)], 1)
                      for ky in range(3)], 1)
    return {"y": _leaky(_conv64(x, w) + b), "dx": _conv64(dy, w.flip(1, 2).permute(3, 1, 2, 0)), "dw": dw,
            "db": g.sum(0)}


def _exact_upsample(case, seed):
    x0, base = (t.to(torch.float64) for t in _upsample_inputs(case, seed))
    z = np.load(WEIGHTS)
    w = {k[2:]: torch.from_numpy(z[k]).cuda().to(torch.bfloat16).to(torch.float64) for k in z if k.startswith("w.")}
    b = {k[2:]: torch.from_numpy(z[k]).cuda().to(torch.float64) for k in z if k.startswith("b.")}
    F = torch.nn.functional
    conv = lambda name, x: _leaky(_conv64(x, w[name]) + b[name])  # noqa: E731
    pool = lambda x: F.avg_pool2d(x.permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1)  # noqa: E731
    up = lambda x: x.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    e1 = conv("enc1b", conv("enc1a", x0))
    e2 = conv("enc2b", conv("enc2a", pool(e1)))
    b2 = conv("botb", conv("bota", pool(e2)))
    d2 = conv("dec2b", conv("dec2a", torch.cat([up(b2), e2], -1)))
    d1 = conv("dec1b", conv("dec1a", torch.cat([up(d2), e1], -1)))
    f = _conv64(d1, w["head"]) + b["head"]
    n, h, wd, _ = f.shape
    f = f.reshape(n, h, wd, 2, 2, 4).permute(0, 1, 3, 2, 4, 5).reshape(n, 2 * h, 2 * wd, 4)
    big = F.interpolate(base.permute(0, 3, 1, 2), scale_factor=2, mode="bilinear", align_corners=False)
    return f + big.permute(0, 2, 3, 1)
