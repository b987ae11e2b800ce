"""The tensor-core maps with the corners' factors made by the map's own CTAs, and by the preparation, at the edges of the rule
between them and of the rounds of 256 corners by 16 (or 8) rows the map's CTAs work in. The F32 map of bytes, which goes through
the FP16 one, is the F32 plane's bit for bit; the BF16 and FP16 maps are within 0.02 and 0.005 of it, the roundings of their
operands (2^-9 and 2^-12 a product, as the configuration's test bounds them), and a near-blank window scores exactly 0."""
import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,tw,th,step,corners", [
    (400, 120, 64, 64, 1, (256, 16)),     # one round, one tile
    (400, 120, 64, 64, 1, (257, 17)),     # a round of one corner, a tile of one row
    (400, 120, 64, 64, 1, (1, 1)),
    (640, 130, 64, 66, 2, (513, 33)),     # three rounds
    (420, 190, 128, 128, 1, (256, 8)),    # eight-row tiles
    (420, 190, 128, 128, 2, (259, 9)),
    (300, 150, 112, 100, 1, (180, 40)),   # the widest template of sixteen-row tiles: the most shared memory
    (900, 90, 64, 64, 1, (768, 20)),      # past what the tensor core hides: the preparation's
    (1100, 120, 96, 96, 1, (1000, 20)),   # four rounds
    (1200, 880, 64, 64, 1, (1025, 801)),  # two tiles across, over 100 tiles
])
def test_maps_whichever_makes_the_factors(vtg_lib, ctx, w, h, tw, th, step, corners):
    import torch

    frame = S.noise_frame(w, h, seed=w + th)
    frame[h // 2:, w // 2:] = 60  # near-blank windows
    patch = S.noise_frame(w, h, seed=w + th)[8:8 + th, 5:5 + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h, 128, 128)
    s.template(app, float(np.sum(app.astype(np.float64) ** 2)))
    win = (3, 3 + corners[0] - 1, 2, 2 + corners[1] - 1)
    assert win[1] + tw < w - 1 and win[3] + th < h - 1
    want = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, *win, step, want_map=True)
    got = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, *win, step, want_map=True)
    assert got[0] == want[0]
    for a, b in zip(got[1:], want[1:]):
        assert a.tobytes() == b.tobytes()
    for prec, tol in ((vtg_lib.NCC_BF16, 0.02), (vtg_lib.NCC_FP16, 0.005)):
        _, v, _, _ = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, *win, step, prec, want_map=True)
        assert np.abs(v - want[1]).max() <= tol
        assert (v[want[1] == 0.0] == 0.0).all()
    s.close()
