"""A search whose tensor-core map gave up in a bounded wait: a device caller's record says so (ntop -1, no score), a host caller gets
VTG_ETIMEOUT, and the searches after it are whole, whoever asked for the one that failed. The checked build ends a map that way
on request, once all its waits have ended, so nothing runs out on the GPU."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WORKLOAD = r"""
import ctypes as C, json, sys
sys.path[:0] = [%(pkg)r]
import numpy as np, torch
import vtg, vtg_synth as S

L = vtg.lib()
ctx = vtg.Context(0)
w, h = 400, 300
frame = S.noise_frame(w, h, seed=5)
patch = frame[40:104, 50:114].astype(np.float32)
app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
d = torch.from_numpy(frame).cuda()
f32 = d.float()
rec = torch.zeros(8, dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
s = vtg.Search(ctx, w, h)
s.template(app, float(np.sum(app.astype(np.float64) ** 2)))

def host(prec, plane=None):
    f = vtg.Found()
    rc = L.vtg_search_run(s.h, d.data_ptr() if plane is None else plane.data_ptr(), w, h, w, vtg.PLANE_U8 if plane is None else vtg.PLANE_F32,
                          1, w, 1, h, 1, prec, C.byref(f), None, None, None, vtg.HOST, None)
    return [rc, f.hx, f.hy, f.ntop]

def device(prec):
    rc = L.vtg_search_run(s.h, d.data_ptr(), w, h, w, vtg.PLANE_U8, 1, w, 1, h, 1, prec, C.cast(rec.data_ptr(), C.POINTER(vtg.Found)), None, None, None,
                          vtg.DEVICE, None)
    ctx.sync()
    r = rec.cpu().numpy()
    v = r.view(np.float32)
    return [rc, int(r[0]), int(r[1]), int(r[6]), float(v[2]), float(v[3])]

out = []
for prec in (vtg.NCC_F32, vtg.NCC_BF16, vtg.NCC_FP16):
    before = host(prec)
    assert L.vtg_check_give_up(1) == 1
    failed = device(prec)
    assert L.vtg_check_give_up(0) == 1
    after = host(prec)
    assert L.vtg_check_give_up(1) == 1
    failed_host = host(prec)
    floats = host(vtg.NCC_F32, f32)  # its map has no such waits
    assert L.vtg_check_give_up(0) == 1
    out.append([before, failed, after, failed_host, floats, device(prec)])
print(json.dumps(out))
"""


def test_a_map_that_gave_up_is_its_own_search_alone(vtg_lib):
    import vtg_build

    assert vtg_lib.lib().vtg_check_give_up(1) == 0
    env = dict(os.environ, VTG_LIB=vtg_build.build(checked=True))
    r = subprocess.run([sys.executable, "-c", WORKLOAD % {"pkg": os.path.join(ROOT, "intel-phi-visiontrack_gb300")}], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    for before, failed, after, failed_host, floats, last in json.loads(r.stdout.strip().splitlines()[-1]):
        assert before[:3] == [0, 100, 80] and before[3] == 8
        assert failed == [0, 0, 0, -1, -2.0, -2.0]
        assert after == before
        assert failed_host[0] == vtg_lib.ETIMEOUT and failed_host[3] == -1
        assert floats == before
        assert last[:4] == before
