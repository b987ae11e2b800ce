"""GPU parity for the pyramid under tk_build's input steps at the edges of its launch's 128 x 64 blocks (level 0 and the halos
of levels 1 to 3 in one launch), inside a batched step with frames that have no steps too, and over more levels than the launch
makes. Bit for bit against the oracle, the -0 of the stretch included."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [1, 2, 3])
@pytest.mark.parametrize("w,h,levels,pad,kind", [
    (32, 32, 1, 0, "low"),
    (33, 47, 3, 5, "warp"),
    (128, 64, 4, 0, "low"),     # one block
    (129, 65, 4, 1, "dark"),    # one pixel more each way
    (416, 272, 4, 0, "warp"),   # blocks inside the frame
    (401, 257, 6, 7, "low"),    # and levels past the launch's
    (200, 150, 4, 0, "flat"),
])
def test_levels_match_the_oracle(vtg_lib, ctx, w, h, levels, pad, kind, opts):
    import torch

    f = S.build_frame(kind, w, h, seed=w + h)
    buf = np.zeros((h, w + pad), np.uint8)
    buf[:, :w] = f
    d = torch.from_numpy(buf).cuda()
    torch.cuda.synchronize()
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=levels))
    plain = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=levels))
    t.set_build(opts)
    t.build(0, d.data_ptr(), stride=w + pad, where=vtg_lib.DEVICE)
    ref = O.pyramid(f, levels, opts=opts)
    for L in range(levels):
        assert t.level(0, L).tobytes() == ref[L].tobytes(), L
    # a step of both trackers: the one without steps keeps its plain pyramid
    b = vtg_lib.Batch(ctx, 2)
    b.prepare(0, [t, plain], [d.data_ptr(), d.data_ptr()], [1, 1], strides=[w + pad, w + pad])
    b.launch(0)
    ctx.sync()
    base = O.pyramid(f, levels)
    for L in range(levels):
        assert t.level(1, L).tobytes() == ref[L].tobytes() and plain.level(1, L).tobytes() == base[L].tobytes(), L
    b.close()
    t.close()
    plain.close()
