"""GPU parity for corner detection where its launches and its selection change form: regions of a whole number of cell rows,
one row, more than 2,048 rows; more candidates than are kept; many equal scores (a lattice: whole blocks of ties, settled in
scan order); spacings from none to most of the region. The corners equal the oracle's, in order."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


def _lattice(w, h, period):
    """Bright squares at a fixed period: corners with one response everywhere inside."""
    y, x = np.mgrid[0:h, 0:w]
    return np.where((x % period < period // 2) & (y % period < period // 2), 200, 60).astype(np.uint8)


@pytest.mark.parametrize("kind,w,h,rect,margin,n,dist,quality", [
    ("noise", 640, 480, (16, 16, 320, 160), 0, 256, 6.0, 0.02),   # a whole number of cell rows
    ("noise", 640, 480, (100, 77, 300, 1), 4, 64, 3.0, 0.02),     # one row: nothing inside
    ("noise", 640, 480, (100, 77, 300, 3), 4, 64, 3.0, 0.02),     # one candidate row
    ("noise", 1920, 1080, (0, 0, 1920, 1080), 12, 512, 4.0, 0.0), # over 8,192 candidates
    ("noise", 640, 480, (0, 0, 640, 480), 5, 512, 0.0, 0.01),     # no spacing: the best 512
    ("noise", 640, 480, (0, 0, 640, 480), 5, 512, 300.0, 0.01),   # few corners fit: every candidate is looked at
    ("noise", 80, 2200, (0, 0, 80, 2200), 3, 200, 5.0, 0.02),     # tall: the rows' counts scanned by themselves
    ("lattice", 800, 600, (0, 0, 800, 600), 8, 512, 9.0, 0.1),    # thousands of equal scores
    ("lattice", 800, 600, (0, 0, 800, 600), 8, 100, 400.0, 0.1),
    ("flat", 200, 150, (0, 0, 200, 150), 2, 100, 5.0, 0.1),
])
def test_corners_are_the_oracles(vtg_lib, ctx, kind, w, h, rect, margin, n, dist, quality):
    import torch

    f = {"noise": lambda: S.noise_frame(w, h, seed=h), "lattice": lambda: _lattice(w, h, 12),
         "flat": lambda: np.full((h, w), 90, np.uint8)}[kind]()
    plane = O.pyramid(f, 1)[0]
    d = torch.from_numpy(plane).cuda()
    torch.cuda.synchronize()
    det = vtg_lib.Detector(ctx, w, h)
    for _ in range(2):  # and again: the detector's state between detections
        xs, ys = det.detect(d.data_ptr(), w, h, w, *rect, margin, n, dist, quality)
        oxs, oys = O.detect(plane, *rect, margin, n, dist, quality)
        assert np.array_equal(xs, oxs) and np.array_equal(ys, oys)
    det.close()
