"""The walk's two launch shapes, for few points and for many, at the line between them (8 points on each of 152 SMs): every point
and cell is walked by one warp with the same operations in either, so the results are the same bit for bit."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pw,ph", [(21, 21), (15, 15), (9, 13), (29, 31)])
@pytest.mark.parametrize("cols,rows", [(38, 32), (39, 32), (35, 33), (3, 5), (38, 1)])
def test_few_and_many_agree(vtg_lib, ctx, pw, ph, cols, rows):
    w, h = max(16 * cols, 64), max(8 * rows, 64)
    f0, f1, _, _ = S.warp_pair(w, h, (1.5, -0.75), 0.5, seed=cols)
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=2, patch_w=pw, patch_h=ph))
    t.build(0, f0)
    t.build(1, f1)
    n = t.cols * t.rows
    cells, lk = t.cells(0, 1)
    mx, my = pw // 2 + 2, ph // 2 + 2
    i = np.arange(n)
    xs = np.clip(i % t.cols * 16 + 8, mx, w - 1 - mx).astype(np.float32)
    ys = np.clip(i // t.cols * 8 + 4, my, h - 1 - my).astype(np.float32)
    reps = -(-1217 // n)
    many = t.points(0, 1, np.tile(xs, reps)[:max(n, 1217)], np.tile(ys, reps)[:max(n, 1217)])
    few = t.points(0, 1, xs[:1216], ys[:1216])
    assert many[:n].tobytes() == lk.tobytes()
    assert many[:len(few)].tobytes() == few.tobytes()
    one = t.points(0, 1, xs[n - 1:], ys[n - 1:])
    assert one.tobytes() == lk[n - 1:].tobytes()
    ref = O.lk_points(O.pyramid(f0, 2), O.pyramid(f1, 2), 1, O.lk_cfg(pw, ph), xs, ys, max_fb=0.5, mode=O.F64)
    ok = (ref["status"] == 0) & (lk["status"] == 0)
    assert (ref["status"] == lk["status"]).mean() >= 0.99
    assert np.abs(np.stack([ref["x"] - lk["x"], ref["y"] - lk["y"]]))[:, ok].max(initial=0) <= 0.01
    t.close()
