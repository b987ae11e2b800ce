"""GPU parity for the F32 appearance search over the forms its maps take: templates much wider than tall over most of the
plane, where the window sums come from the integral images and the column sums' room would be longer than the
template."""
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
