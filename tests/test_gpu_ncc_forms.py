"""GPU parity for the F32 appearance search over the forms its maps take. An 8-bit plane and the same values as an F32 plane
have the same maps, bit for bit, whichever way an 8-bit plane's map is made (large templates and windows go through the FP16
tensor-core filter): over tile edges, template widths, windows, and pictures with ties and flat parts. Templates much wider
than tall over most of the plane take their window sums from the integral images, where the column sums' room would be longer
than the template."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


def _template(frame, x, y, tw, th):
    patch = frame[y:y + th, x:x + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    return app, float(np.sum(app.astype(np.float64) ** 2))


@pytest.mark.parametrize("w,h,tw,th,step", [(217, 300, 96, 52, 2), (300, 200, 128, 33, 1), (301, 187, 128, 47, 2)])
def test_wide_templates_over_the_plane(vtg_lib, ctx, w, h, tw, th, step):
    import torch

    frame = S.noise_frame(w, h, seed=33)
    app, norm = _template(frame, 31, 57, tw, th)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h)
    s.template(app, norm)
    a, av, ax, ay = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, 1, w, 1, h, step, want_map=True)
    b, bv, bx, by = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, 1, w, 1, h, step, want_map=True)
    s.close()
    ref, rv, _, _ = O.search_slot(frame.astype(np.float32), app, norm, 1, w, 1, h, step, mode=O.F64)
    assert a == b and np.array_equal(av, bv) and np.array_equal(ax, bx) and np.array_equal(ay, by)
    assert np.abs(av - rv[:a["cells"]]).max() < 1e-4
    assert (a["hx"], a["hy"]) == (ref["hx"], ref["hy"]) and abs(a["ncc"] - ref["ncc"]) < 1e-4


def _picture(kind, w, h):
    f = S.noise_frame(w, h, seed=w + h)
    if kind == "stripes":  # every row the same: ties down each column of corners
        f = np.ascontiguousarray(np.broadcast_to(f[:1], (h, w)))
    elif kind == "half flat":  # near-blank windows score exactly 0
        f[h // 2:] = 90
    elif kind == "dim":  # low contrast, far from mid grey
        f = (f // 16 + 3).astype(np.uint8)
    return f


@pytest.mark.parametrize("kind", ["noise", "stripes", "half flat", "dim"])
@pytest.mark.parametrize("w,h,tw,th,step,win", [
    (1100, 90, 32, 64, 1, None),                # past one tile of 1,024 corners
    (1057, 121, 32, 64, 1, (1, 1024, 1, 33)),   # exactly one tile wide, two and a row of 16 high
    (400, 200, 128, 17, 1, None),               # eight-row tiles, four whole steps of columns
    (300, 190, 104, 33, 2, (7, 250, 9, 130)),   # a part step, every second corner, a window inside
    (190, 170, 64, 33, 1, (60, 60, 20, 20)),    # one corner
    (641, 481, 24, 40, 1, None),                # a small template over a large window
    (64, 140, 48, 48, 1, None),                 # the narrowest plane
    (1300, 800, 16, 16, 1, None),               # the F32 plane's map in CTAs of 32 corner rows (over 608 of them)
    (330, 250, 72, 40, 2, None),                # and where a window is wider than its CTA's threads
])
def test_bytes_and_floats_have_one_map(vtg_lib, ctx, kind, w, h, tw, th, step, win):
    import torch

    frame = _picture(kind, w, h)
    app, norm = _template(S.noise_frame(w, h, seed=w + h) if kind != "dim" else frame, 5, 8, tw, th)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h)
    s.template(app, norm)
    x0, x1, y0, y1 = win or (1, w, 1, h)
    a, av, ax, ay = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, x0, x1, y0, y1, step, want_map=True)
    b, bv, bx, by = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, x0, x1, y0, y1, step, want_map=True)
    s.close()
    assert a["cells"] > 0 and a == b
    assert np.array_equal(av.view(np.uint32), bv.view(np.uint32)) and np.array_equal(ax, bx) and np.array_equal(ay, by)
