"""The still picture's vectors, walked two cells a warp, against the tracker's one cell a warp with the same settings: the same
operations on the same pixels, so the same bits. Grids with an odd number of columns, rows past the last CTA's, the smallest
picture, and cells of one warp that end differently: flat, changed, moved out of reach and tracked ones side by side."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(32, 32), (33, 47), (48, 40), (80, 200), (333, 101), (640, 472)])
@pytest.mark.parametrize("scene", ["shift", "mixed", "noise", "flat"])
def test_vectors_match_the_cells_kernel(vtg_lib, ctx, w, h, scene):
    import torch

    rng = np.random.default_rng(w + h)
    f0, f1, _, _ = S.warp_pair(w, h, (1.25, -0.5), 0.5, seed=w)
    if scene == "mixed":  # 12-pixel blocks, not the cells': flat in both, replaced, far away, or as they are
        for y in range(0, h, 12):
            for x in range(0, w, 12):
                k = rng.integers(4)
                b0, b1 = f0[y:y + 12, x:x + 12], f1[y:y + 12, x:x + 12]
                if k == 0:
                    b0[:] = b1[:] = 90
                elif k == 1:
                    b1[:] = rng.integers(0, 256, b1.shape)
                elif k == 2:
                    b1[:] = np.roll(b1, 5, axis=1)
    elif scene == "noise":
        f0, f1 = (rng.integers(0, 256, (h, w)).astype(np.uint8) for _ in range(2))
    elif scene == "flat":
        f0[:] = 77
        f1[:] = 78
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=1, patch_w=15, patch_h=15, max_iter=6, max_residual=16.0, fb_max=0.25,
                                            cell_w=16, cell_h=8))
    t.build(0, f0)
    t.build(1, f1)
    want, _ = t.cells(0, 1)
    st = vtg_lib.Still(ctx, w, h)
    planes = [torch.from_numpy(O.pyramid(f, 1)[0]).cuda() for f in (f0, f1)]
    torch.cuda.synchronize()
    for p in planes:
        st.frame(p.data_ptr(), w)
    got, _, _ = st.read()
    assert len(got) == len(want)
    for k in ("u", "v", "diff", "sigma"):
        assert got[k].tobytes() == want[k].tobytes(), k
    assert np.array_equal(got["state"] & 0xff, want["state"] & 0xff)
    st.close()
    t.close()
