"""GPU parity for frame generation at the edges of its launches' blocks: 64 x 32 blocks of the field's first level and the
three levels under it, tiles of 16 pixels eight to a CTA, fields of one and of few blocks, two to seven levels. Bit for
bit against the oracle, on a device buffer and inside the generator."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,shift,kind", [
    (64, 64, (3.0, -2.0), "pair"),        # two levels: the scene test launches by itself
    (65, 97, (-4.0, 5.0), "pair"),
    (128, 130, (0.0, 0.0), "pair"),       # one block wide, ragged by one row; no motion
    (257, 131, (20.0, -15.0), "pair"),    # vectors past the borders
    (400, 333, (-9.0, 7.0), "pair"),      # blocks inside and on the edges
    (272, 264, (0.0, 0.0), "scene"),      # every field zero
    (2300, 2100, (11.0, 6.0), "pair"),    # seven levels: three launches for the pyramid
])
def test_sizes_match_the_oracle(vtg_lib, ctx, w, h, shift, kind):
    import torch

    f0, f1 = S.framegen_pair(kind, w, h, shift, seed=w + h)
    p0, p1 = O.pyramid(f0, 1)[0], O.pyramid(f1, 1)[0]
    a, b = torch.from_numpy(p0).cuda(), torch.from_numpy(p1).cuda()
    torch.cuda.synchronize()
    fg = vtg_lib.Framegen(ctx, w, h)
    pic = fg.run(a.data_ptr(), w, b.data_ptr(), w)
    r = fg.fields()
    fg.close()
    o = O.framegen(p0, p1)
    assert r["scene"] == (kind == "scene")
    for key in ("raw", "fil", "up"):
        for L, (x, y) in enumerate(zip(r[key], o[key])):
            assert x.tobytes() == y.tobytes(), (key, L)
    assert r["mid"].tobytes() == o["mid"].tobytes() and np.array_equal(pic, o["pic"])
