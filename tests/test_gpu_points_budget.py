"""A context's budget bounds what its trackers hold between calls: host point lists keep no scratch there. Without a budget they do, and
vtg_ctx_held counts it. The lists' results are the same."""
import ctypes as C

import numpy as np
import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_lists_under_a_budget_keep_nothing(vtg_lib):
    import torch

    w, h, n = 200, 160, 16384
    cfg = vtg_lib.config(w, h, levels=2)
    one = vtg_lib.lib().vtg_tracker_bytes(C.byref(cfg))
    f0, f1, _, _ = S.warp_pair(w, h, (1.5, -0.75), 0.5, seed=9)
    rng = np.random.default_rng(2)
    xs, ys = (rng.uniform(10, m - 10, n).astype(np.float32) for m in (w, h))
    outs = []
    for budget in (0, 8 * one):
        c = vtg_lib.Context(0, hbm_budget=budget)
        ts = [vtg_lib.Tracker(c, cfg) for _ in range(8)]
        for t in ts:
            t.build(0, f0)
            t.build(1, f1)
        c.sync()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for t in ts:
            outs.append(t.points(0, 1, xs, ys).tobytes())
        torch.cuda.synchronize()
        grown = free - torch.cuda.mem_get_info()[0]
        assert c.used() == 8 * one
        if budget:
            assert c.held() == 8 * one and grown <= 0
        else:
            assert c.held() - 8 * one == 8 * 2 * n * 48 and grown >= 8 * MB
        for t in ts:
            t.close()
        assert c.used() == c.held() == 0
        c.close()
    assert len(set(outs)) == 1
