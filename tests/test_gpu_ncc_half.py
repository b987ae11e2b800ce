"""The half-pixel pass at the edges of its row groups (four rows a warp, 32 a CTA) and column groups (1, 2 or 4 a lane), bytes
and floats: the position of the FP64 oracle's search and its score within 1e-4."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1, 2])
@pytest.mark.parametrize("tw,th", [(8, 40), (32, 31), (40, 33), (64, 32), (72, 65), (128, 17)])
def test_half_pixel_corners(vtg_lib, ctx, tw, th, step):
    import torch

    w, h = 260, 170
    frame = S.noise_frame(w, h, seed=tw)
    moved = S.bilinear(frame.astype(np.float64), np.arange(w)[None, :] + 0.5 + 0 * np.arange(h)[:, None], np.arange(h)[:, None] + 0.0 * np.arange(w)[None, :])
    patch = moved[60:60 + th, 50:50 + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    norm = float(np.sum(app.astype(np.float64) ** 2))
    ref, _, _, _ = O.search_slot(frame.astype(np.float32), app, norm, 1, w, 1, h, step, mode=O.F64)
    u8, f32 = torch.from_numpy(frame).cuda(), torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h, 128, 128)
    s.template(app, norm)
    a = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, 1, w, 1, h, step)
    b = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, 1, w, 1, h, step)
    s.close()
    for f in (a, b):
        assert (f["hx"], f["hy"]) == (ref["hx"], ref["hy"]) == (101, 120) and abs(f["ncc"] - ref["ncc"]) < 1e-4
