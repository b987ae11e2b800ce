"""Calls right behind a caller's kernel that releases its dependents at its start and writes their input a little later (0.1 ms): a
point list in device memory, and a still picture's frame, are read only once they are written."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CYCLES = 200_000


@pytest.fixture(scope="module")
def late(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("early") / "early_release.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "c", "early_release.cu")], check=True)
    f = C.CDLL(so).early_release
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_longlong, C.c_void_p]

    def write(out, src, stream):
        assert f(out.data_ptr(), src.data_ptr(), src.numel(), CYCLES, stream) == 0

    return write


@pytest.mark.parametrize("n", [200, 3000])
def test_point_lists(vtg_lib, ctx, late, n):
    import torch

    w, h = 320, 240
    f0, f1, _, _ = S.warp_pair(w, h, (1.5, -0.75), 0.5, seed=9)
    t = vtg_lib.Tracker(ctx, vtg_lib.config(w, h, levels=3))
    t.build(0, f0)
    t.build(1, f1)
    rng = np.random.default_rng(n)
    lists = [np.stack([rng.uniform(20, m - 20, n) for m in (w, h)]).astype(np.float32) for _ in range(3)]
    want = [t.points(0, 1, p[0], p[1]) for p in lists]
    src = [torch.from_numpy(p).cuda() for p in lists]
    xy = torch.zeros((2, n), device="cuda")
    out = torch.zeros((n, 32), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for k in range(12):
        late(xy, src[k % 3], t.stream)
        assert vtg_lib.lib().vtg_points(t.h, 0, 1, 2, n, xy.data_ptr(), xy.data_ptr() + 4 * n, None, None, out.data_ptr(), vtg_lib.DEVICE,
                                        None) == 0
        t.sync()
        assert out.cpu().numpy().tobytes() == want[k % 3].tobytes(), k
    t.close()


def test_still_frames(vtg_lib, ctx, late):
    import torch

    w, h = 320, 200
    rng = np.random.default_rng(5)
    base = S.noise_frame(w, h, seed=w).astype(int)
    src = [torch.from_numpy(O.pyramid(np.clip(base + rng.integers(-3, 4, base.shape), 0, 255).astype(np.uint8), 1)[0]).cuda()
           for _ in range(8)]
    cur = torch.zeros((h, w), device="cuda")
    a, b = vtg_lib.Still(ctx, w, h, 4, 1.0, 40.0), vtg_lib.Still(ctx, w, h, 4, 1.0, 40.0)
    torch.cuda.synchronize()
    for f in src:
        a.frame(f.data_ptr(), w)
        late(cur, f, b.stream())
        b.frame(cur.data_ptr(), w)
        ctx.sync()
        for p, q in zip(a.read(), b.read()):
            assert p.tobytes() == q.tobytes()
    a.close()
    b.close()
