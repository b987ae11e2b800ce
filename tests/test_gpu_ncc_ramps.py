"""F32 searches of bytes on pictures where the filter rules little or nothing out (ramps: every window is its neighbours' plus a
constant, so a cell's corners tie to within the filter's bound): the map is the F32 plane's bit for bit on either side of the list's
length from which every corner is scored, and such a search takes no longer than the direct map and the filter together."""
import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu


def _ramp(w, h, share, steep):
    y, x = np.mgrid[0:h, 0:w]
    r = (x + y) % 256 if steep else (3 * x + 2 * y) // 16 % 256
    return np.where(x < w * share, r, S.noise_frame(w, h, seed=w)).astype(np.uint8)


def _search(vtg_lib, ctx, frame, tw, th):
    import torch

    patch = frame[3:3 + th, 2:2 + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, frame.shape[1], frame.shape[0], 128, 128)
    s.template(app, float(np.sum(app.astype(np.float64) ** 2)))
    return s, u8, f32


@pytest.mark.parametrize("share", [0.2, 0.35, 0.5, 1.0])
@pytest.mark.parametrize("w,h,tw,th,step,win,steep", [
    (420, 300, 64, 64, 1, None, True),
    (420, 300, 64, 64, 2, None, True),
    (421, 303, 96, 96, 1, None, False),           # ragged cells and blocks
    (421, 303, 104, 72, 2, (3, 250, 2, 190), False),
    (300, 260, 128, 128, 1, None, False),         # one block a CTA in shared memory
    (330, 280, 128, 128, 2, None, False),
    (400, 300, 64, 64, 1, (5, 44, 3, 20), True),  # two blocks for 304 places
    (900, 500, 32, 24, 1, None, True),            # a small template over a large window
    (700, 460, 40, 40, 1, None, True),            # a part step of columns
])
def test_ramps_have_the_direct_map(vtg_lib, ctx, w, h, tw, th, step, win, steep, share):
    frame = _ramp(w, h, share, steep)
    s, u8, f32 = _search(vtg_lib, ctx, frame, tw, th)
    win = win or (1, w, 1, h)
    a = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, *win, step, want_map=True)
    b = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, *win, step, want_map=True)
    s.close()
    assert a[0]["cells"] > 0 and a[0] == b[0]
    for p, q in zip(a[1:], b[1:]):
        assert p.tobytes() == q.tobytes()


@pytest.mark.parametrize("size", [96, 128])
def test_a_ramp_takes_no_longer_than_the_direct_map_and_the_filter(vtg_lib, ctx, size):
    w, h = 1920, 1080
    frame = _ramp(w, h, 1.0, False)
    s, u8, f32 = _search(vtg_lib, ctx, frame, size, size)
    _, t8 = s.profile(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, 1, w, 1, h, 1, vtg_lib.NCC_F32, 5)
    _, t32 = s.profile(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, 1, w, 1, h, 1, vtg_lib.NCC_F32, 5)
    s.close()
    assert t8 < 1.5 * t32, (t8, t32)  # a list of every corner took 2.5 to 3 times
