"""Scores at and below -2, which a norm smaller than the template's own gives: a cell with nothing above -2 keeps -2 and its origin,
in the map of bytes (by the FP16 filter, whose candidates reach a little under -2) as in the F32 plane's, bit for bit."""
import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1, 2])
@pytest.mark.parametrize("share", [0.25, 0.24999, 0.2499, 0.249, 0.1])
@pytest.mark.parametrize("tw,th,corners", [(64, 64, (1, 1)), (64, 64, (1, 20)), (96, 96, (40, 3))])
def test_cells_with_nothing_above_the_floor(vtg_lib, ctx, tw, th, corners, share, step):
    import torch

    w, h, x, y = 300, 250, 37, 21
    frame = S.noise_frame(w, h, seed=tw)
    patch = frame[y:y + th, x:x + tw].astype(np.float32)
    app = (np.float32(patch.mean(dtype=np.float64)) - patch).astype(np.float32)  # the negative of what is there
    norm = float(np.sum(app.astype(np.float64) ** 2)) * share                    # so its score there is -1 / sqrt(share)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h)
    s.template(app, norm)
    win = (x, x + corners[0] - 1, y, y + corners[1] - 1)
    a = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, *win, step, want_map=True)
    b = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, *win, step, want_map=True)
    s.close()
    assert a[0] == b[0]
    for p, q in zip(a[1:], b[1:]):
        assert p.tobytes() == q.tobytes()
    if corners == (1, 1) and share < 0.24999:
        assert a[1][0] == -2.0 and a[0]["ntop"] == 0
