"""F32 searches of bytes that go through the FP16 tensor-core filter, over pictures with ties, flat parts, little contrast and a mean far
from the middle grey (the filter's bound is loosest there): the map is the F32 plane's bit for bit. Shapes at the edges of tiles,
template widths with a part step of columns, windows inside. Which searches take the filter is checked too, by the checked build,
whose filter gives up on request."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# w, h, tw, th, step, window
FILTERED = [
    (1100, 150, 64, 64, 1, None),               # past one tile of 1,024 corners
    (1090, 99, 64, 64, 1, (1, 1024, 1, 33)),    # exactly one tile wide, two and a row of 16 high
    (420, 230, 128, 33, 1, None),               # eight-row tiles
    (330, 220, 104, 40, 2, (7, 217, 9, 150)),   # a part step, every second corner, a window inside
    (260, 170, 64, 64, 1, (60, 60, 20, 20)),    # one corner
    (300, 300, 40, 104, 1, None),               # part steps in the second of two
    (300, 300, 48, 96, 1, None),
    (300, 260, 56, 80, 2, None),
    (300, 300, 72, 72, 1, None),                # and in the third
    (280, 290, 128, 128, 2, None),
    (620, 480, 32, 40, 1, None),                # a small template over a large window
    (256, 200, 64, 64, 1, None),
]
DIRECT = [
    (620, 480, 32, 40, 1, (1, 300, 1, 300)),    # the same over a smaller one
    (120, 300, 64, 64, 1, None),                # too narrow: a row of bounds takes 1,024 places, of some four a plane's pixel
    (300, 300, 64, 64, 4, None),                 # step 4
]


def _picture(kind, w, h):
    f = S.noise_frame(w, h, seed=w + h)
    if kind == "stripes":  # every row the same: ties down each column of corners
        f = np.ascontiguousarray(np.broadcast_to(f[:1], (h, w)))
    elif kind == "half flat":  # near-blank windows score exactly 0
        f[h // 2:] = 90
    elif kind == "dim":  # little contrast, a mean of some eleven
        f = (f // 16 + 3).astype(np.uint8)
    elif kind == "bright":  # and of some 250
        f = np.clip(np.random.default_rng(w).normal(250, 1.5, (h, w)), 0, 255).astype(np.uint8)
    elif kind == "binary":
        f = (np.random.default_rng(h).integers(0, 2, (h, w)) * 255).astype(np.uint8)
    return f


def _template(frame, tw, th, spike=None):
    patch = frame[8:8 + th, 5:5 + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    if spike:
        app[th // 2, tw // 2] = spike
    return app, float(np.sum(app.astype(np.float64) ** 2))


def _both(vtg_lib, ctx, frame, app, norm, win, step):
    import torch

    h, w = frame.shape
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h)
    s.template(app, norm)
    win = win or (1, w, 1, h)
    a = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, *win, step, want_map=True)
    b = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, *win, step, want_map=True)
    s.close()
    assert a[0]["cells"] > 0 and a[0] == b[0]
    for p, q in zip(a[1:], b[1:]):
        assert p.tobytes() == q.tobytes()


@pytest.mark.parametrize("kind", ["noise", "stripes", "half flat", "dim", "bright", "binary"])
@pytest.mark.parametrize("w,h,tw,th,step,win", FILTERED)
def test_the_filtered_map_is_the_direct_one(vtg_lib, ctx, kind, w, h, tw, th, step, win):
    frame = _picture(kind, w, h)
    app, norm = _template(frame, tw, th)
    if norm > 0:
        _both(vtg_lib, ctx, frame, app, norm, win, step)


WORKLOAD = r"""
import ctypes as C, json, sys
sys.path[:0] = [%(pkg)r, %(tests)r]
import numpy as np, torch
import vtg, test_gpu_ncc_filter as T

ctx = vtg.Context(0)
out = []
assert vtg.lib().vtg_check_give_up(1) == 1
for spike, shapes in ((None, T.FILTERED), (None, T.DIRECT), (7e4, T.FILTERED)):
    got = []
    for w, h, tw, th, step, win in shapes:
        frame = T._picture("noise", w, h)
        app, norm = T._template(frame, tw, th, spike)
        d = torch.from_numpy(frame).cuda()
        torch.cuda.synchronize()
        s = vtg.Search(ctx, w, h)
        s.template(app, norm)
        f = vtg.Found()
        x0, x1, y0, y1 = win or (1, w, 1, h)
        got.append(vtg.lib().vtg_search_run(s.h, d.data_ptr(), w, h, w, vtg.PLANE_U8, x0, x1, y0, y1, step, vtg.NCC_F32, C.byref(f), None,
                                            None, None, vtg.HOST, None))
        s.close()
    out.append(got)
print(json.dumps(out))
"""


def test_which_searches_take_the_filter(vtg_lib):
    import vtg_build

    env = dict(os.environ, VTG_LIB=vtg_build.build(checked=True))
    code = WORKLOAD % {"pkg": os.path.join(ROOT, "intel-phi-visiontrack_gb300"), "tests": os.path.join(ROOT, "tests")}
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    filtered, direct, spiked = json.loads(r.stdout.strip().splitlines()[-1])
    assert filtered == [vtg_lib.ETIMEOUT] * len(FILTERED)
    assert direct == [vtg_lib.OK] * len(DIRECT) and spiked == [vtg_lib.OK] * len(FILTERED)
