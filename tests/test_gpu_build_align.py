"""The builds' byte loads, plain and under the input steps, at every alignment of the frame's first byte and of its rows (sixteen bytes from shifted words, whole
vectors or single bytes), with guard bytes around the frame that a wrong one would take for its minimum or maximum. Bit for bit
against the oracle."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [0, 1, 2, 3])
@pytest.mark.parametrize("w,h,start,pad", [(275, 130, 1, 0), (275, 130, 2, 2), (275, 130, 3, 13), (272, 130, 16, 0), (272, 130, 4, 4),
                                           (290, 90, 7, 1), (51, 70, 5, 0), (35, 33, 1, 2), (34, 33, 0, 0)])
def test_any_alignment(vtg_lib, ctx, w, h, start, pad, opts):
    import torch

    f = np.clip(S.build_frame("warp", w, h, seed=w), 20, 230)
    n = start + h * (w + pad) + 16
    buf = np.where(np.arange(n) % 2 == 0, 0, 255).astype(np.uint8)
    rows = np.lib.stride_tricks.as_strided(buf[start:], (h, w), (w + pad, 1))
    rows[:] = f
    d = torch.from_numpy(buf).cuda()
    torch.cuda.synchronize()
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=3))
    t.set_build(opts)
    t.build(0, d.data_ptr() + start, stride=w + pad, where=vtg_lib.DEVICE)
    ref = O.pyramid(np.ascontiguousarray(f), 3, opts=opts)
    for L in range(3):
        assert t.level(0, L).tobytes() == ref[L].tobytes(), L
    t.close()
