"""Host point lists longer than any before, whose device scratch has to grow, while another stream of the device is busy: the call
does not wait for that stream, and the lists before and after give what they give alone."""
import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu


def test_growing_lists_wait_for_no_other_stream(vtg_lib, ctx):
    import torch

    w, h = 320, 240
    f0, f1, _, _ = S.warp_pair(w, h, (1.5, -0.75), 0.5, seed=9)
    rng = np.random.default_rng(2)
    lists = [[torch.from_numpy(rng.uniform(20, m - 20, n).astype(np.float32)).pin_memory() for m in (w, h)]
             for n in (100, 3000, 50, 12000, 16384, 20000)]
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=3))
    alone = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=3))
    for k in (t, alone):
        k.build(0, f0)
        k.build(1, f1)
    ctx.sync()
    busy, done = torch.cuda.Stream(), torch.cuda.Event()
    for xs, ys in lists:
        want = alone.points(0, 1, xs.numpy(), ys.numpy())
        out = torch.zeros((len(xs), 32), dtype=torch.uint8).pin_memory()
        torch.cuda.synchronize()
        with torch.cuda.stream(busy):
            torch.cuda._sleep(400_000_000)  # 0.2 s at 2 GHz
            done.record(busy)
        assert vtg_lib.lib().vtg_points(t.h, 0, 1, 2, len(xs), xs.data_ptr(), ys.data_ptr(), None, None, out.data_ptr(),
                                        vtg_lib.HOST, None) == 0
        assert not done.query(), len(xs)
        t.sync()
        assert out.numpy().tobytes() == want.tobytes()
    t.close()
    alone.close()
