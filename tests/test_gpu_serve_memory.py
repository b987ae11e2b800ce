"""The served loop's limit bounds the device memory that its trackers hold, not only the bytes they are charged: in a context without
a budget a tracker may hold more than its charge (rows at a fixed pitch), and a limited loop keeps to compact trackers unless all
its streams fit the limit as they would be held. Device memory is read while the loop runs."""
import ctypes as C
import threading
import time

import pytest

import vtg_synth as S

pytestmark = pytest.mark.gpu

W, H, N = 640, 480, 16
MB = 1 << 20


def _bytes(vtg_lib):
    return vtg_lib.lib().vtg_tracker_bytes(C.byref(vtg_lib.config(W, H, levels=4)))


def _run(vtg_lib, ctx, budget):
    """(stats, the most device memory in use during the run less what was before it, the streams' last cells)"""
    import numpy as np
    import torch

    f0, f1, _, _ = S.warp_pair(W, H, (1.5, -0.75), 0.5, seed=3)
    bufs = [torch.from_numpy(f).pin_memory() for f in (f0, f1)] * N
    streams = [dict(width=W, height=H, fps=60.0, start_s=0.0, frames=12) for _ in range(N)]
    last = [np.zeros((W // 16) * (H // 8), vtg_lib.CELL_DTYPE) for _ in range(N)]
    most, stop = [0], threading.Event()
    before = torch.cuda.mem_get_info()[0]

    def watch():
        while not stop.is_set():
            most[0] = max(most[0], before - torch.cuda.mem_get_info()[0])
            time.sleep(0.002)

    t = threading.Thread(target=watch)
    t.start()
    try:
        st = vtg_lib.serve(ctx, streams, [b.data_ptr() for b in bufs], vtg_lib.config(64, 64, levels=4), duration_s=1.0, max_batch=16,
                           hbm_budget=budget, last_cells=last)
    finally:
        stop.set()
        t.join()
    return st, most[0], b"".join(x.tobytes() for x in last)


def test_a_limited_loop_holds_its_limit(vtg_lib):
    import torch

    ctx = vtg_lib.Context(0)
    one = _bytes(vtg_lib)
    _run(vtg_lib, ctx, 0)  # the modules are loaded, the pools made
    torch.cuda.synchronize()
    free, free_most, free_cells = _run(vtg_lib, ctx, 0)
    limited, most, cells = _run(vtg_lib, ctx, N * one)
    assert free["served"] == limited["served"] == 12 * N
    assert limited["streams_admitted"] == N and limited["streams_waited"] == 0
    assert free_most > 2 * N * one  # the run that has no limit does hold the padding
    # 2 MB granules, and what is not the streams' trackers: two batches' tables and the results' staging
    assert most <= N * (one + 2 * MB) + 16 * MB, (most, N * one)
    assert cells == free_cells
    ctx.close()


def test_a_limit_with_room_changes_nothing(vtg_lib):
    ctx = vtg_lib.Context(0)
    one = _bytes(vtg_lib)
    used = ctx.used()
    t = vtg_lib.Tracker(ctx, vtg_lib.config(W, H, levels=4))
    held = ctx.held()
    t.close()
    assert ctx.used() == used == 0 == ctx.held() and held > 2 * one
    _run(vtg_lib, ctx, 0)
    st, most, _ = _run(vtg_lib, ctx, N * held)
    assert st["served"] == 12 * N and 2 * N * one < most <= N * (held + 2 * MB) + 16 * MB
    ctx.close()
