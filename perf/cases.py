"""Timed cases of the sparse tracking path: the calls that a program around this library makes for each frame, through
the Python binding (and, where results stay on the GPU, the C ABI behind it).

A case is a dict of plain values; ``kind`` says which call it stands for:

* ``pyramid``: ``Tracker.build`` of a frame that is on the GPU, with tk_build's optional input steps;
* ``pair``: one camera's frame: ``build``, then the per-cell flow from the frame before it; ``host`` says whether the
  frame comes from and the cells go to host memory (one camera served by itself) or stay on the GPU;
* ``points``: the feature list's flow, host arrays in and out;
* ``batch``: one step of many cameras, a captured graph replayed, results copied to GPU buffers;
* ``search``: the appearance search of a lost region, on a frame's bytes or on a tracker's level 1;
* ``detect``: corners of a region of a tracker's level 0;
* ``still``: one frame of the still picture;
* ``framegen``: one frame generated between two.

Frames are blurred uniform noise (sigma 1.5 px) and the same scene moved by a shift and a smooth field, the benchmark's
own scenes, made on the GPU. ``exact`` restates each computation in 64 bits with torch alone.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "intel-phi-visiontrack_gb300"))
import vtg  # noqa: E402

LK = dict(patch=21, max_iter=10, eps=0.01, min_eig=0.1, max_residual=25.0, fb_max=0.5)  # vtg.config's defaults
STILL_LK = dict(patch=15, max_iter=6, eps=0.01, min_eig=0.1, max_residual=16.0, fb_max=0.25)
APP_W, APP_H = 32, 21  # the reference's template
MARGIN = 12            # seed_at's distance from the plane's edges


def listed():
    return [
        # the smallest call: one VGA camera's pyramid, no options
        dict(name="pyramid_vga", kind="pyramid", w=640, h=480, levels=3, opts=0, pad=0),
        # a ragged frame in a wider buffer, with the contrast stretch and the pre-gauss (a dim camera)
        dict(name="pyramid_options_719p", kind="pyramid", w=1281, h=719, levels=4, opts=3, pad=23),
        # one VGA camera served by itself: upload, pyramid, 1,200 cells, results on the host (latency)
        dict(name="pair_vga_host", kind="pair", w=640, h=480, levels=3, cell_w=16, cell_h=16, flow_level=0, host=True),
        # one 1080p camera, everything on the GPU: 16,200 cells a frame
        dict(name="pair_1080p", kind="pair", w=1920, h=1080, levels=4, cell_w=16, cell_h=8, flow_level=0, host=False),
        # a tracker's feature list: 512 points, host arrays (OP_LK)
        dict(name="points_512", kind="points", w=1920, h=1080, levels=4, n=512, guess=False),
        # eight 1080p cameras in one step, the served loop's full batch
        dict(name="batch_8x1080p", kind="batch", w=1920, h=1080, levels=4, n=8, mixed=False),
        # a lost region looked for over the whole level 1, every second corner, as the served loop asks for it
        dict(name="search_level1_f32", kind="search", w=1920, h=1080, tw=APP_W, th=APP_H, step=2, precision=0, level1=True),
        # reacquisition over a whole 1080p frame with exact products, the default precision
        dict(name="search_64_f32", kind="search", w=1920, h=1080, tw=64, th=64, step=1, precision=0, level1=False),
        # the same with a large template and BF16 products
        dict(name="search_96_bf16", kind="search", w=1920, h=1080, tw=96, th=96, step=1, precision=1, level1=False),
        # reseeding a region's features (seed_at): 128 corners of a box
        dict(name="detect_box", kind="detect", w=1920, h=1080, rx=700.5, ry=400.25, rw=384.0, rh=307.0, n=128, dist=8.0,
             quality=0.05),
        # a still 1080p camera's frame
        dict(name="still_1080p", kind="still", w=1920, h=1080, avg=8),
        # a frame between two 1080p frames
        dict(name="framegen_1080p", kind="framegen", w=1920, h=1080),
    ]


def _size(rng, wmin, wmax):
    """A frame's size: its width over the logarithm of the range, odd or even, a height between 9/16 and 3/4 of it."""
    w = int(round(math.exp(rng.uniform(math.log(wmin), math.log(wmax)))))
    return w, max(64, int(w * rng.uniform(0.5625, 0.75)))


def draw(rng: random.Random):
    kind = rng.choice(["pyramid", "pair", "points", "batch", "search", "search", "detect", "still", "framegen"])
    if kind == "pyramid":
        w, h = _size(rng, 320, 3840)
        return dict(kind=kind, w=w, h=h, levels=rng.randint(1, 5), opts=rng.choice([0, 0, 1, 2, 3]), pad=rng.choice([0, 0, 7, 64]))
    if kind == "pair":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, levels=rng.randint(2, 4), cell_w=16, cell_h=rng.choice([8, 16]),
                    flow_level=rng.choice([0, 0, 1]), host=rng.random() < 0.5)
    if kind == "points":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, levels=rng.randint(2, 4), n=int(math.exp(rng.uniform(math.log(16), math.log(2048)))),
                    guess=rng.random() < 0.5)
    if kind == "batch":
        w, h = _size(rng, 320, 1280)
        return dict(kind=kind, w=w, h=h, levels=rng.randint(3, 4), n=rng.randint(2, 12), mixed=rng.random() < 0.7)
    if kind == "search":
        w, h = _size(rng, 320, 1920)
        if rng.random() < 0.3:
            return dict(kind=kind, w=max(w, 400), h=max(h, 240), tw=APP_W, th=APP_H, step=rng.choice([1, 2]), precision=0, level1=True)
        step = rng.choice([1, 1, 2])  # every second corner: the smaller templates, as in a tracker's own searches
        return dict(kind=kind, w=w, h=h, tw=8 * rng.randint(2, 12 if step == 1 else 8), th=rng.randint(12, 96 if step == 1 else 64),
                    step=step, precision=rng.choice([0, 1, 2]), level1=False)
    if kind == "detect":
        w, h = _size(rng, 320, 1920)
        rw, rh = w * rng.uniform(0.1, 1.0), h * rng.uniform(0.15, 1.0)
        return dict(kind=kind, w=w, h=h, rx=round((w - rw) * rng.random(), 2), ry=round((h - rh) * rng.random(), 2), rw=round(rw, 2),
                    rh=round(rh, 2), n=rng.randint(32, 512), dist=float(rng.randint(4, 16)), quality=rng.choice([0.01, 0.05, 0.1]))
    if kind == "still":
        w, h = _size(rng, 320, 1920)
        return dict(kind=kind, w=w, h=h, avg=rng.randint(2, 32))
    w, h = _size(rng, 320, 1920)
    return dict(kind=kind, w=w, h=h)


# ---------------------------------------------------------------- inputs

def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + k)


def _blur(a):
    """Gaussian, sigma 1.5, eleven taps, clamped borders, along the last axis."""
    taps = [math.exp(-k * k / 4.5) for k in range(-5, 6)]
    n = a.shape[-1]
    at = torch.arange(n, device=a.device)
    return sum((t / sum(taps)) * a[..., (at + k - 5).clamp(0, n - 1)] for k, t in enumerate(taps))


def _scene(w, h, seed, k=0):
    """A picture's continuous values, float32 (h, w)."""
    noise = torch.randint(0, 256, (h, w), generator=_gen(seed, k), device="cuda").float()
    return _blur(_blur(noise).t().contiguous()).t().contiguous()


def _moved(img, seed, k, shift, amp):
    """img moved by a shift and a smooth field of amplitude amp: a bilinear resample at x - d(x, y)."""
    h, w = img.shape
    grid = torch.rand((1, 2, 6, 8), generator=_gen(seed, 100 + k), device="cuda") * 2 - 1
    field = torch.nn.functional.interpolate(grid, size=(h, w), mode="bicubic", align_corners=True)[0].clamp(-1, 1) * amp
    y, x = torch.meshgrid(torch.arange(h, device="cuda").float(), torch.arange(w, device="cuda").float(), indexing="ij")
    x = (x - shift[0] - field[0]).clamp(0, w - 1)
    y = (y - shift[1] - field[1]).clamp(0, h - 1)
    xi, yi = x.floor().clamp(max=w - 2).long(), y.floor().clamp(max=h - 2).long()
    fx, fy = x - xi, y - yi
    top = img[yi, xi] + fx * (img[yi, xi + 1] - img[yi, xi])
    bot = img[yi + 1, xi] + fx * (img[yi + 1, xi + 1] - img[yi + 1, xi])
    return top + fy * (bot - top)


def _u8(img):
    return (img + 0.5).floor().clamp(0, 255).to(torch.uint8).contiguous()


def _pair_frames(w, h, seed, k=0, amp=0.5):
    r = random.Random(int(seed) * 7919 + k)
    shift = (r.uniform(-6, 6), r.uniform(-6, 6))
    base = _scene(w, h, seed, k)
    return _u8(base), _u8(_moved(base, seed, k, shift, amp))


def _option_frame(c, seed):
    """A dim frame (what the stretch is for) in rows of w + pad bytes."""
    f = _u8(_scene(c["w"], c["h"], seed))
    if c["opts"] & 1:
        f = (100 + (f.int() * 40) // 255).to(torch.uint8)
    buf = torch.zeros((c["h"], c["w"] + c["pad"]), dtype=torch.uint8, device="cuda")
    buf[:, :c["w"]] = f
    return buf


def _points(c, seed):
    g = np.random.default_rng(int(seed))
    xs = g.uniform(20.0, c["w"] - 20.0, c["n"]).astype(np.float32)
    ys = g.uniform(20.0, c["h"] - 20.0, c["n"]).astype(np.float32)
    if not c["guess"]:
        return xs, ys, None, None
    return xs, ys, g.uniform(-2, 2, c["n"]).astype(np.float32), g.uniform(-2, 2, c["n"]).astype(np.float32)


def _template(frame, c, seed):
    """A template cut from the frame, its gain, offset and noise changed: zero-mean floats and the sum of squares."""
    r = random.Random(int(seed) * 31 + 7)
    h, w = frame.shape
    x, y = r.randint(2, w - c["tw"] - 4), r.randint(2, h - c["th"] - 4)
    patch = frame[y:y + c["th"], x:x + c["tw"]].float()
    noise = torch.randn(patch.shape, generator=_gen(seed, 55), device="cuda") * 3
    patch = (patch * r.uniform(0.8, 1.2) + r.uniform(-20, 20) + noise).round().clamp(0, 255).double()
    app = (patch - patch.mean()).float()
    return app.cpu().numpy(), float(np.float32((app.double() ** 2).sum().item()))


def _still_frames(c, seed):
    """A still camera: the scene drifting a little, sensor noise, a textured square moving through."""
    base = _scene(c["w"], c["h"], seed)
    tex = _scene(48, 48, seed, 9) * 0.5 + 100.0
    out = []
    for i in range(6):
        img = _moved(base, seed, 0, (0.03 * i, 0.02 * i), 0.0)
        x0 = min(c["w"] // 5 + 3 * i, c["w"] - 48)
        img[c["h"] // 3:c["h"] // 3 + 48, x0:x0 + 48] = tex
        img = img + torch.rand(img.shape, generator=_gen(seed, 300 + i), device="cuda") * 6.0 - 3.0
        out.append(_u8(img).float() * 64.0)
    return out


class _DevicePlane:
    """An F32 plane in device memory that a library object owns, as torch sees it; it keeps that object."""

    def __init__(self, owner, ptr, w, h, pitch):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (h, w), "strides": (4 * pitch, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _level(t, s, level):
    p, w, h, pitch = vtg.level_device(t, s, level)
    return torch.as_tensor(_DevicePlane(t, p, w, h, pitch), device="cuda")


def _batch_sizes(c):
    half = ((c["w"] // 2) | 1, (c["h"] // 2) | 1)
    return [half if c["mixed"] and j % 2 else (c["w"], c["h"]) for j in range(c["n"])]


def prepare(c, seed):
    kind, w, h = c["kind"], c["w"], c["h"]
    ctx = vtg.Context(0)
    s = dict(kind=kind, ctx=ctx, case=c, k=0)
    if kind == "pyramid":
        s["frame"] = _option_frame(c, seed)
        s["t"] = t = vtg.Tracker(ctx, vtg.config(w, h, levels=c["levels"]))
        t.set_build(c["opts"])
        s["levels"] = [_level(t, 0, L) for L in range(c["levels"])]
    elif kind in ("pair", "points"):
        f0, f1 = _pair_frames(w, h, seed)
        if kind == "pair":
            s["t"] = t = vtg.Tracker(ctx, vtg.config(w, h, levels=c["levels"], cell_w=c["cell_w"], cell_h=c["cell_h"],
                                                    flow_level=c["flow_level"]))
            n = t.cols * t.rows
            if c["host"]:
                s["pinned"] = [f.cpu().pin_memory() for f in (f0, f1)]
                s["frames"] = [p.numpy() for p in s["pinned"]]
            else:
                s["frames"] = [f0, f1]
                s["cells"] = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
                s["lk"] = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
        else:
            s["t"] = t = vtg.Tracker(ctx, vtg.config(w, h, levels=c["levels"]))
            s["points"] = _points(c, seed)
        torch.cuda.synchronize()
        t.build(0, f0.data_ptr(), where=vtg.DEVICE)
        if kind == "points":
            t.build(1, f1.data_ptr(), where=vtg.DEVICE)
        t.sync()
    elif kind == "batch":
        sizes = _batch_sizes(c)
        s["frames"] = [_pair_frames(a, b, seed, j) for j, (a, b) in enumerate(sizes)]
        s["ts"] = [vtg.Tracker(ctx, vtg.config(a, b, levels=c["levels"])) for a, b in sizes]
        s["cells"] = [torch.zeros((t.cols * t.rows, 6), dtype=torch.int32, device="cuda") for t in s["ts"]]
        torch.cuda.synchronize()
        for t, (f0, _) in zip(s["ts"], s["frames"]):
            t.build(0, f0.data_ptr(), where=vtg.DEVICE)
            t.sync()
        s["b"] = b = vtg.Batch(ctx, c["n"])
        for slot in (0, 1):  # slot 0 takes the second frames into set 1, slot 1 the first ones into set 0
            b.prepare(slot, s["ts"], [f[1 - slot].data_ptr() for f in s["frames"]], [1 - slot] * c["n"])
            b.capture(slot)
        s["stream"] = b.stream
    elif kind == "search":
        f0, f1 = _pair_frames(w, h, seed)
        if c["level1"]:
            s["t"] = t = vtg.Tracker(ctx, vtg.config(w, h, levels=2))
            torch.cuda.synchronize()
            t.build(0, f0.data_ptr(), where=vtg.DEVICE)
            t.build(1, f1.data_ptr(), where=vtg.DEVICE)
            a = t.store_appearance(0, *_region(c, seed))
            app, norm = a["pix"], float(a["norm"])
            s["plane"] = vtg.level_device(t, 1, 1) + (vtg.PLANE_F32,)
        else:
            app, norm = _template(f0, c, seed)
            s["frame"] = f1
            s["plane"] = (f1.data_ptr(), w, h, w, vtg.PLANE_U8)
        s["search"] = vtg.Search(ctx, s["plane"][1], s["plane"][2], 128, 128)
        torch.cuda.synchronize()
        s["search"].template(app, norm)
    elif kind == "detect":
        f = _u8(_scene(w, h, seed))
        s["t"] = t = vtg.Tracker(ctx, vtg.config(w, h, levels=1))
        s["det"] = vtg.Detector(ctx, w, h)
        torch.cuda.synchronize()
        t.build(0, f.data_ptr(), where=vtg.DEVICE)
        t.sync()
        s["plane"] = vtg.level_device(t, 0, 0)
    elif kind == "still":
        s["frames"] = _still_frames(c, seed)
        s["still"] = st = vtg.Still(ctx, w, h, c["avg"], 1.0, 4.0)
        s["cells"] = torch.zeros((st.cols * st.rows, 6), dtype=torch.int32, device="cuda")
        s["motion"] = torch.zeros(12, dtype=torch.int32, device="cuda")
        p, pitch = ctypes.c_void_p(), ctypes.c_int()
        vtg.check(vtg.lib().vtg_still_mean(st.h, ctypes.byref(p), ctypes.byref(pitch)), "vtg_still_mean")
        s["mean"] = torch.as_tensor(_DevicePlane(st, p.value, w, h, pitch.value), device="cuda")
        torch.cuda.synchronize()
        for f in s["frames"][:2]:
            st.frame(f.data_ptr(), w)
        s["k"] = 2
    else:
        f0, f1 = _pair_frames(w, h, seed, amp=3.0)
        s["frames"] = [f0.float() * 64.0, f1.float() * 64.0]
        s["fg"] = fg = vtg.Framegen(ctx, w, h)
        p, pitch = fg.frame_ptr()
        s["out"] = torch.as_tensor(_DevicePlane(fg, p, w, h, pitch), device="cuda")
    torch.cuda.synchronize()
    return s


def _region(c, seed):
    r = random.Random(int(seed) * 13 + 1)
    return r.uniform(90.0, c["w"] - 90.0), r.uniform(70.0, c["h"] - 70.0), 70.0, 50.0  # level 1's template fits it


def _cells_out(a):
    f = a.view(torch.float32)
    return dict(u=f[:, 0], v=f[:, 1], diff=f[:, 2], state=a[:, 3], sigma=f[:, 4])


def _lk_out(a):
    f = a.view(torch.float32)
    return dict(x=f[:, 0], y=f[:, 1], min_eig=f[:, 2], residual=f[:, 3], cov=f[:, 4:7], iters_status=a[:, 7])


def _lk_host(a):
    return dict(x=a["x"], y=a["y"], min_eig=a["min_eig"], residual=a["residual"],
                cov=[a["cov_xx"], a["cov_xy"], a["cov_yy"]], iters=a["iters"].view("<i2"), status=a["status"].view("<i2"))


def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "pyramid":
        s["t"].build(0, s["frame"].data_ptr(), stride=c["w"] + c["pad"], where=vtg.DEVICE)
        return s["levels"]
    if kind == "pair":
        t, cur = s["t"], (s["k"] + 1) & 1
        s["k"] += 1
        if c["host"]:
            t.build(cur, s["frames"][cur])
            cells, lk = t.cells(1 - cur, cur)
            return dict(u=cells["u"], v=cells["v"], diff=cells["diff"], state=cells["state"].view("<i4"), sigma=cells["sigma"],
                        lk=_lk_host(lk))
        t.build(cur, s["frames"][cur].data_ptr(), where=vtg.DEVICE)
        t.cells_device(1 - cur, cur, s["cells"].data_ptr(), s["lk"].data_ptr())
        return dict(_cells_out(s["cells"]), lk=_lk_out(s["lk"]))
    if kind == "points":
        xs, ys, gx, gy = s["points"]
        return _lk_host(s["t"].points(0, 1, xs, ys, gx, gy))
    if kind == "batch":
        s["b"].replay(s["k"] & 1)
        s["k"] += 1
        for t, buf in zip(s["ts"], s["cells"]):
            vtg.check(vtg.lib().vtg_tracker_results(t.h, buf.data_ptr(), None, vtg.DEVICE, s["stream"]), "vtg_tracker_results")
        return [_cells_out(x) for x in s["cells"]]
    if kind == "search":
        p, w, h, pitch, typ = s["plane"]
        return s["search"].run(p, w, h, pitch, typ, 1, w, 1, h, c["step"], c["precision"])
    if kind == "detect":
        p, w, h, pitch = s["plane"]
        return list(s["det"].detect(p, w, h, pitch, c["rx"], c["ry"], c["rw"], c["rh"], MARGIN, c["n"], c["dist"], c["quality"]))
    if kind == "still":
        f = s["frames"][s["k"] % len(s["frames"])]
        s["k"] += 1
        s["still"].frame(f.data_ptr(), c["w"])
        vtg.check(vtg.lib().vtg_still_read(s["still"].h, s["cells"].data_ptr(), s["motion"].data_ptr(), None, 0, vtg.DEVICE, None),
                  "vtg_still_read")
        return dict(_cells_out(s["cells"]), counts=s["motion"][:4], drift=s["motion"].view(torch.float32)[4:10], mean=s["mean"])
    a, b = s["frames"]
    s["fg"].run(a.data_ptr(), c["w"], b.data_ptr(), c["w"], pic=False)
    return s["out"]


# ---------------------------------------------------------------- the work a pass cannot do without

def _pyr_values(w, h, levels):
    n = 0
    for _ in range(levels):
        n += w * h
        w, h = (w + 1) // 2, (h + 1) // 2
    return n


def _lk_flops(n, levels, p, iters=4.4):
    """Both walks of n points: a template build and (measured on the scenes above) 4.4 iterations a level, and a
    residual pass, in the reference's operation counts."""
    a = p["patch"] ** 2
    return n * 2 * (levels * (9 * (p["patch"] + 2) ** 2 + 20 * a + iters * 14 * a) + 12 * a)


def work(c):
    kind, w, h = c["kind"], c["w"], c["h"]
    if kind == "pyramid":
        v = _pyr_values(w, h, c["levels"])
        return dict(bytes=w * h + 4 * v, flops=8 * v)
    if kind == "pair":
        fw, fh = -(-w // 2 ** c["flow_level"]), -(-h // 2 ** c["flow_level"])
        n = -(-fw // c["cell_w"]) * -(-fh // c["cell_h"])
        v = _pyr_values(w, h, c["levels"])
        return dict(bytes=w * h + 8 * v + 56 * n, flops=8 * v + _lk_flops(n, c["levels"] - c["flow_level"], LK))
    if kind == "points":
        return dict(bytes=c["n"] * (48 + 2 * 4 * 24 * 24 * c["levels"]), flops=_lk_flops(c["n"], c["levels"], LK))
    if kind == "batch":
        b = f = 0
        for x, y in _batch_sizes(c):
            n, v = -(-x // 16) * -(-y // 8), _pyr_values(x, y, c["levels"])
            b += x * y + 8 * v + 24 * n
            f += 8 * v + _lk_flops(n, c["levels"], LK)
        return dict(bytes=b, flops=f)
    if kind == "search":
        if c["level1"]:
            w, h = (w + 1) // 2, (h + 1) // 2
        corners = max(0, w - c["tw"] - 2) * max(0, h - c["th"] - 2) / c["step"] ** 2
        return dict(bytes=w * h * (4 if c["level1"] else 1) + 4 * c["tw"] * c["th"], flops=2 * corners * c["tw"] * c["th"])
    if kind == "detect":
        return dict(bytes=4 * c["rw"] * c["rh"] + 8 * c["n"], flops=60 * c["rw"] * c["rh"])
    if kind == "still":
        n = -(-w // 16) * -(-h // 8)
        return dict(bytes=12 * w * h + 24 * n, flops=2 * w * h + _lk_flops(n, 1, STILL_LK))
    # the two frames in, the frame out; the search's 256 offsets of 64 pixels a block on every level
    v = _pyr_values((w + 1) // 2, (h + 1) // 2, 6)
    return dict(bytes=12 * w * h + 8 * v, flops=2 * 256 * v + 14 * w * h)


# ---------------------------------------------------------------- the same in 64 bits, by torch alone

def _reduce(p, half=128.0, scale=256.0):
    """img_reduce of a Q6 plane: the 5 x 5 binomial at every second pixel, clamped borders, floor((sum + 128) / 256)."""
    for _ in range(2):
        n = p.shape[-1]
        at = 2 * torch.arange((n + 1) // 2, device=p.device)
        p = sum(k * p[..., (at + i - 2).clamp(0, n - 1)] for i, k in enumerate((1, 4, 6, 4, 1))).t()
    return ((p + half) / scale).floor()


def _pyramid(level0, levels):
    out = [level0]
    while len(out) < levels:
        out.append(_reduce(out[-1]))
    return out


def _build(c, seed):
    f = _option_frame(c, seed)[:, :c["w"]].double() * 64.0
    if c["opts"] & 1:
        lo, hi = f.min().item(), f.max().item()
        gain = 16320.0 / (hi - lo) if hi > lo else 1.0
        f = (f * gain - lo * gain).round().clamp(0, 16320)
    if c["opts"] & 2:
        for _ in range(2):
            at = torch.arange(f.shape[-1], device=f.device)
            f = sum(k * f[..., (at + i - 2).clamp(0, f.shape[-1] - 1)] for i, k in enumerate((1, 4, 6, 4, 1))).t()
        f = ((f + 128) / 256).floor()
    return _pyramid(f, c["levels"])


def _window(p, x, y, half, n):
    """Bilinear samples of p at (x + i, y + j), i, j = -half .. n - half - 1: (points, n, n)."""
    xi, yi = x.floor(), y.floor()
    fx, fy = (x - xi)[:, None, None], (y - yi)[:, None, None]
    k = torch.arange(n + 1, device=p.device) - half
    cx = (xi.long()[:, None] + k).clamp(0, p.shape[1] - 1)
    cy = (yi.long()[:, None] + k).clamp(0, p.shape[0] - 1)
    a = p[cy[:, :, None], cx[:, None, :]]
    a = a[:, :, :-1] + fx * (a[:, :, 1:] - a[:, :, :-1])
    return a[:, :-1] + fy * (a[:, 1:] - a[:, :-1])


def _track(I, J, x, y, gx, gy, q):
    """One walk down the pyramid for every point at once (lk_driver.inc)."""
    n, P, dev = len(x), q["patch"], x.device
    half, m, area = P // 2, P // 2 + 1, P * P
    gx, gy = gx / 2 ** (len(I) - 1), gy / 2 ** (len(I) - 1)
    zero = torch.zeros(n, dtype=torch.float64, device=dev)
    status, iters = torch.zeros(n, dtype=torch.long, device=dev), torch.zeros(n, dtype=torch.long, device=dev)
    eig0, valid0 = zero.clone(), torch.zeros(n, dtype=torch.bool, device=dev)
    last = None

    def inside(p, px, py):
        return (px >= m) & (py >= m) & (px < p.shape[1] - m - 1) & (py < p.shape[0] - m - 1)

    for L in range(len(I) - 1, -1, -1):
        px, py = x / 2 ** L, y / 2 ** L
        live = inside(I[L], px, py)
        if L == 0:
            status |= torch.where(live, 0, 1)
        s = _window(I[L], px, py, half + 1, P + 2)
        dx, dy = s[:, :, 2:] - s[:, :, :-2], s[:, 2:] - s[:, :-2]
        tx = (2 * dx[:, 1:-1] + dx[:, :-2] + dx[:, 2:]) / 512
        ty = (2 * dy[:, :, 1:-1] + dy[:, :, :-2] + dy[:, :, 2:]) / 512
        T = s[:, 1:-1, 1:-1]
        gxx, gxy, gyy = (tx * tx).sum((1, 2)), (tx * ty).sum((1, 2)), (ty * ty).sum((1, 2))
        det = gxx * gyy - gxy * gxy
        lmax = 0.5 * (gxx + gyy + ((gxx - gyy) ** 2 + 4 * gxy * gxy).sqrt())
        eig = torch.where(lmax > 0, det / (lmax * area), zero)
        if L == 0:
            eig0 = torch.where(live, eig, zero)
        low = (eig < q["min_eig"]) | (det <= 0)
        if L == 0:
            status |= torch.where(live & low, 2, 0)
        live = live & ~low
        if L == 0:
            valid0 = live.clone()
        idet = torch.where(live, 1 / det, zero)
        vx, vy, going = zero.clone(), zero.clone(), live.clone()
        for _ in range(q["max_iter"]):
            qx, qy = px + gx + vx, py + gy + vy
            ok = inside(J[L], qx, qy)
            if L == 0:
                status |= torch.where(going & ~ok, 1, 0)
                valid0 &= ~(going & ~ok)
            going = going & ok
            if not bool(going.any()):
                break
            d = T - _window(J[L], torch.where(going, qx, px), torch.where(going, qy, py), half, P)
            bx, by = (d * tx).sum((1, 2)), (d * ty).sum((1, 2))
            ex = torch.where(going, (gyy * bx - gxy * by) * idet / 64, zero)
            ey = torch.where(going, (gxx * by - gxy * bx) * idet / 64, zero)
            vx, vy, iters = vx + ex, vy + ey, iters + going.long()
            going = going & (ex * ex + ey * ey >= q["eps"] ** 2)
        gx, gy = gx + vx, gy + vy
        if L:
            gx, gy = 2 * gx, 2 * gy
        else:
            last = (T, gxx, gxy, gyy, idet)
    good = valid0 & (status == 0)
    ok = inside(J[0], x + gx, y + gy)
    status |= torch.where(good & ~ok, 1, 0)
    good = good & ok
    T, gxx, gxy, gyy, idet = last
    d = (T - _window(J[0], torch.where(good, x + gx, x), torch.where(good, y + gy, y), half, P)) / 64
    res = torch.where(good, d.abs().sum((1, 2)) / area, zero)
    s2 = torch.where(good, (d * d).sum((1, 2)) / (area - 2), zero)
    status |= torch.where(res > q["max_residual"], 4, 0)
    return dict(x=x + gx, y=y + gy, min_eig=eig0, residual=res, cov_xx=s2 * gyy * idet, cov_xy=-s2 * gxy * idet,
                cov_yy=s2 * gxx * idet, iters=iters, status=status)


def _flow(I, J, x, y, gx, gy, q):
    """lk_track and lk_flowback, some thousands of points at a time."""
    parts = []
    for a in range(0, len(x), 8192):
        k = slice(a, a + 8192)
        o = _track(I, J, x[k], y[k], gx[k], gy[k], q)
        back = _track(J, I, o["x"], o["y"], x[k] - o["x"], y[k] - o["y"], q)
        miss = (back["x"] - x[k]) ** 2 + (back["y"] - y[k]) ** 2
        bad = (o["status"] == 0) & ((back["status"] != 0) | ~(miss <= q["fb_max"] ** 2))
        o["status"] = o["status"] | torch.where(bad, 8, 0)
        parts.append(o)
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def _cells(I, J, cw, ch, q):
    """still_vectors: the flow at every cell's centre and the cells' records, row by row."""
    h, w = I[0].shape
    cols, rows = -(-w // cw), -(-h // ch)
    m = q["patch"] // 2 + 2
    x = (torch.arange(cols, device="cuda").double() * cw + cw // 2).clamp(m, w - 1 - m).repeat(rows)
    y = (torch.arange(rows, device="cuda").double() * ch + ch // 2).clamp(m, h - 1 - m).repeat_interleave(cols)
    o = _flow(I, J, x, y, torch.zeros_like(x), torch.zeros_like(x), q)
    d = (J[0] - I[0]).abs()
    d = torch.cat([d, d[:, -1:].expand(-1, cols * cw - w)], 1)
    count = torch.full((rows,), float(cw * ch), device="cuda", dtype=torch.float64)
    count[-1] = cw * (h - (rows - 1) * ch)
    d = torch.cat([d, torch.zeros((rows * ch - h, cols * cw), device="cuda", dtype=torch.float64)])
    diff = d.reshape(rows, ch, cols, cw).sum((1, 3)) / count[:, None] / 64
    sigma = torch.where(o["status"] == 0, (o["cov_xx"] + o["cov_yy"]).clamp(min=0).sqrt(), torch.zeros_like(x))
    return dict(u=o["x"] - x, v=o["y"] - y, diff=diff.reshape(-1), state=o["status"], sigma=sigma), o


def _still(c, seed):
    """The still picture after the prepared frames and one more: cells, statistics, mean."""
    frames = [f.double() for f in _still_frames(c, seed)]
    h, w = frames[0].shape
    cols, rows = -(-w // 16), -(-h // 8)
    n = cols * rows
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    count, usual, mean = torch.zeros(n, dtype=torch.long, device="cuda"), 0.0, None
    for k in range(3):
        f = frames[k]
        if k == 0:
            cell = dict(u=zero, v=zero, diff=zero, state=torch.zeros(n, dtype=torch.long, device="cuda"), sigma=zero)
        else:
            cell, _ = _cells([mean], [f], 16, 8, STILL_LK)
        hist = torch.bincount((cell["diff"] * 16).long().clamp(max=255), minlength=256).cumsum(0)
        noise = min(255, int((hist < n // 2).sum())) / 16.0
        limit = max(3 * noise, 4.0)
        everything = k >= 2 and noise > max(3 * usual, 4.0)
        if not everything and k >= 1:
            usual = noise if k == 1 else usual + (noise - usual) / 32
        lk = cell["state"]
        own = ((lk == 0) & ((cell["u"] ** 2 + cell["v"] ** 2).sqrt() > (12 * cell["sigma"]).clamp(min=1.0))) | ((lk & 4) != 0) | \
            (cell["diff"] > limit)
        votes = torch.nn.functional.avg_pool2d(own.double().reshape(1, 1, rows, cols), 3, 1, 1).reshape(-1) * 9
        moved = (votes > 1.5) | everything
        count = torch.where(moved, 1, (count + 1).clamp(max=c["avg"]))
        weight = (1.0 / count.double()).reshape(rows, cols).repeat_interleave(8, 0).repeat_interleave(16, 1)[:h, :w]
        mean = f.clone() if mean is None else mean + weight * (f - mean)
        cell["state"] = lk | (own.long() << 8) | (moved.long() << 9) | (count << 16)
        good = (lk == 0) & ~moved
        g = max(1, int(good.sum()))
        mu, mv = cell["u"][good].sum().item() / g, cell["v"][good].sum().item() / g
        var = (cell["u"][good] ** 2 + cell["v"][good] ** 2).sum().item() / g - mu * mu - mv * mv
    counts = torch.tensor([cols, rows, int((lk == 0).sum()), int(moved.sum())])
    drift = torch.tensor([count.double().mean().item(), mu, mv, math.sqrt(max(0.0, var)), noise, limit], dtype=torch.float64)
    return dict(cell, counts=counts, drift=drift, mean=mean)


def _ncc(st, s1, s2, n, norm):
    nvar = n * s2 - s1 * s1
    return torch.where(nvar <= math.floor(n * norm / 16), torch.zeros_like(st), st / (norm * nvar.clamp(min=1) / n).sqrt())


def _search(c, seed):
    f0, f1 = _pair_frames(c["w"], c["h"], seed)
    if c["level1"]:
        cx, cy, _, _ = _region(c, seed)
        plane = _pyramid(f1.double() * 64, 2)[1]
        x, y = int(cx / 2) - APP_W // 2, int(cy / 2) - APP_H // 2
        app = _pyramid(f0.double() * 64, 2)[1][y:y + APP_H, x:x + APP_W]
        app = app - app.mean()
        norm = float((app * app).sum())
    else:
        plane = f1.double()
        a, norm = _template(f0, c, seed)
        app = torch.from_numpy(a).double().cuda()
    h, w = plane.shape
    th, tw = app.shape
    n, st_ = tw * th, c["step"]
    x1, y1 = w - tw - 2, h - th - 2  # corners 1 .. x1, 1 .. y1
    size = [h + th, w + tw]
    corr = torch.fft.irfft2(torch.fft.rfft2(plane - plane.mean(), size) * torch.fft.rfft2(app, size).conj(), size)[:h, :w]
    corr = corr + plane.mean() * app.sum()

    def box(p):
        t = torch.nn.functional.pad(p.cumsum(0).cumsum(1), (1, 0, 1, 0))
        return t[th:, tw:] - t[:-th, tw:] - t[th:, :-tw] + t[:-th, :-tw]

    b1, b2 = box(plane), box(plane * plane)
    v = _ncc(corr[1:y1 + 1, 1:x1 + 1] - plane[1:y1 + 1, 1:x1 + 1] * app.sum(), b1[1:y1 + 1, 1:x1 + 1], b2[1:y1 + 1, 1:x1 + 1], n, norm)
    v = v[::st_, ::st_]
    per = 16 // st_
    cr, cc = (y1 - 1) // 16 + 1, (x1 - 1) // 16 + 1
    v = torch.nn.functional.pad(v, (0, cc * per - v.shape[1], 0, cr * per - v.shape[0]), value=-9.0)
    v = v.reshape(cr, per, cc, per).permute(0, 2, 1, 3).reshape(cr * cc, per * per)
    best, at = v.max(1)
    order = sorted(range(cr * cc), key=lambda i, b=best.tolist(): (-b[i], i))[:8]
    around = 2 * st_ - 1 if st_ > 1 else 1

    def half(hx, hy):
        x, y, ox, oy = hx >> 1, hy >> 1, hx & 1, hy & 1
        if x < 1 or y < 1 or x + tw + 1 >= w - 1 or y + th + 1 >= h - 1:
            return -1.0
        q = sum(plane[y + b:y + b + th, x + a:x + a + tw] for b in (0, oy) for a in (0, ox)) / 4
        return _ncc(((q - plane[y, x]) * app).sum(), q.sum(), (q * q).sum(), n, norm).item()

    found = []
    for i in order:
        k = int(at[i])
        mx, my = 1 + (i % cc) * 16 + (k % per) * st_, 1 + (i // cc) * 16 + (k // per) * st_
        best_half = None
        for b in range(-around, around + 1):
            for a in range(-around, around + 1):
                s = half(2 * mx + a, 2 * my + b)
                if best_half is None or s > best_half[0]:
                    best_half = (s, 2 * mx + a, 2 * my + b)
        found.append(best_half)
    top = max(found, key=lambda f: f[0])
    second = max([f[0] for f in found if (f[1] - top[1]) ** 2 > tw * tw or (f[2] - top[2]) ** 2 > th * th], default=-2.0)

    def parabola(l, m, r):
        den = l - 2 * m + r
        return 0.0 if den >= 0 else min(0.5, max(-0.5, 0.5 * (l - r) / den))

    return dict(hx=top[1], hy=top[2], ncc=top[0], second=second, ntop=len(found), cells=cr * cc,
                ox=parabola(half(top[1] - 1, top[2]), top[0], half(top[1] + 1, top[2])),
                oy=parabola(half(top[1], top[2] - 1), top[0], half(top[1], top[2] + 1)))


def exact(c, seed):
    kind = c["kind"]
    if kind == "pyramid":
        return _build(c, seed)
    if kind in ("pair", "points"):
        I, J = (_pyramid(f.double() * 64, c["levels"]) for f in _pair_frames(c["w"], c["h"], seed))
        if kind == "points":
            xs, ys, gx, gy = (None if a is None else torch.from_numpy(a).double().cuda() for a in _points(c, seed))
            gx, gy = (torch.zeros_like(xs) if a is None else a for a in (gx, gy))
            o = _flow(I, J, xs, ys, gx, gy, LK)
            return dict(x=o["x"], y=o["y"], min_eig=o["min_eig"], residual=o["residual"], cov=[o["cov_xx"], o["cov_xy"], o["cov_yy"]],
                        iters=o["iters"], status=o["status"])
        f = c["flow_level"]
        cells, o = _cells(I[f:], J[f:], c["cell_w"], c["cell_h"], LK)
        lk = dict(x=o["x"], y=o["y"], min_eig=o["min_eig"], residual=o["residual"])
        if c["host"]:
            lk.update(cov=[o["cov_xx"], o["cov_xy"], o["cov_yy"]], iters=o["iters"], status=o["status"])
        else:
            lk.update(cov=torch.stack([o["cov_xx"], o["cov_xy"], o["cov_yy"]], 1), iters_status=o["iters"] | (o["status"] << 16))
        return dict(cells, lk=lk)
    if kind == "batch":
        out = []
        for j, (w, h) in enumerate(_batch_sizes(c)):
            I, J = (_pyramid(f.double() * 64, c["levels"]) for f in _pair_frames(w, h, seed, j))
            out.append(_cells(I, J, 16, 8, LK)[0])
        return out
    if kind == "search":
        return _search(c, seed)
    if kind == "still":
        return _still(c, seed)
    return None  # detect returns places of whole pixels, framegen whole Q6 values: neither is rounded
