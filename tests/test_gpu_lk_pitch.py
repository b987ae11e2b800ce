"""The trackers' two layouts: every level's rows 2,080 floats apart (a context without a budget, frames 256 to 2,080 wide), which
the LK kernels are compiled for, and rows as far apart as each level's width asks. The same operations on the same pixels: the
same bits, for one stream's cells, few and many points, and a batch of either layout or of both; and the same charge."""
import ctypes as C

import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu

WIDE = 2080


def _results(L, t, f0, f1, n):
    t.build(0, f0)
    t.build(1, f1)
    cells, lk = t.cells(0, 1)
    rng = np.random.default_rng(n)
    w, h = f0.shape[1], f0.shape[0]
    xs, ys = (rng.uniform(0, m, n).astype(np.float32) for m in (w, h))
    return cells.tobytes() + lk.tobytes() + t.points(0, 1, xs, ys).tobytes()


@pytest.mark.parametrize("patch", [(21, 21), (15, 15), (9, 13)])
@pytest.mark.parametrize("w,h,levels", [(255, 131, 3), (256, 131, 3), (641, 483, 4), (2048, 96, 2), (2049, 96, 1), (2080, 96, 3),
                                        (2081, 96, 2)])
def test_layouts_agree(vtg_lib, ctx, w, h, levels, patch):
    cfg = vtg_lib.config(w, h, levels=levels, patch_w=patch[0], patch_h=patch[1])
    f0, f1, _, _ = S.warp_pair(w, h, (1.5, -0.75), 0.5, seed=w)
    bytes_ = vtg_lib.lib().vtg_tracker_bytes(C.byref(cfg))
    small = vtg_lib.Context(0, hbm_budget=bytes_)
    out = []
    for c in (ctx, small):
        used = c.used()
        t = vtg_lib.Tracker(c, cfg)
        assert c.used() - used == bytes_
        pitch = [vtg_lib.level_device(t, 0, k)[3] for k in range(levels)]
        assert pitch == ([WIDE] * levels if c is ctx and 256 <= w <= WIDE else [(-(-w // 2 ** k) + 31) & ~31 for k in range(levels)])
        out.append([_results(vtg_lib, t, f0, f1, n) for n in (40, 1300)])
        t.close()
        assert c.used() == used
    assert out[0] == out[1]
    small.close()


@pytest.mark.parametrize("widths", [(320, 500), (200, 230), (320, 200, 500)])
def test_batch_of_either_layout(vtg_lib, ctx, widths):
    import torch

    fs = [S.warp_pair(w, 160, (1.25, 0.5), 0.5, seed=w)[:2] for w in widths]
    ts = [vtg_lib.Tracker(ctx, vtg_lib.config(w, 160, levels=3)) for w in widths]
    d = [torch.from_numpy(f1).cuda() for _, f1 in fs]
    torch.cuda.synchronize()
    want = []
    for t, (f0, f1) in zip(ts, fs):
        t.build(0, f0)
        t.build(1, f1)
        cells, lk = t.cells(0, 1)
        want.append(cells.tobytes() + lk.tobytes())
    b = vtg_lib.Batch(ctx, len(ts))
    b.prepare(0, ts, [x.data_ptr() for x in d], [1] * len(ts))
    b.launch(0)
    ctx.sync()
    for t, x in zip(ts, want):
        cells, lk = vtg_lib.tracker_results(t)
        assert cells.tobytes() + lk.tobytes() == x
    b.close()
    for t in ts:
        t.close()
