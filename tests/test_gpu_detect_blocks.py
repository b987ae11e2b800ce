"""GPU parity for the corner selection over many blocks: a spacing wide enough that the corners run out long before their number
is reached, so that every candidate kept is looked at, 1,024 at a time, against lists of taken corners of very different
lengths. The corners equal the oracle's, in order, each time. The first case is one in which a lane that came late out of those
lists had its warp leave the walk early."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


def _bytes(w, h, seed):
    return np.random.default_rng(seed).integers(0, 256, (h, w)).astype(np.uint8)


@pytest.mark.parametrize("kind,w,h,seed,rect,margin,n,dist,quality", [
    ("noise", 1456, 693, 933724, (485.33519, -6.7453864, 1179.3107, 645.41545), 2, 256, 40.0, 0.01),
    ("noise", 1456, 693, 7, (0, 0, 1456, 693), 0, 512, 30.0, 0.0),
    ("noise", 1456, 693, 8, (0, 0, 1456, 693), 0, 512, 57.0, 0.0),
    ("noise", 1200, 900, 9, (33.5, 40.25, 1100, 800), 8, 256, 90.0, 0.01),
    ("bytes", 800, 600, 10, (0, 0, 800, 600), 4, 512, 24.0, 0.0),
    ("bytes", 800, 600, 11, (0, 0, 800, 600), 4, 512, 33.3, 0.0),
    ("bytes", 640, 480, 12, (10, 10, 600, 450), 4, 100, 40.0, 0.0),
    ("noise", 640, 480, 13, (0, 0, 640, 480), 2, 512, 27.0, 0.0),
])
def test_corners_of_many_blocks(vtg_lib, ctx, kind, w, h, seed, rect, margin, n, dist, quality):
    import torch

    plane = O.pyramid(_bytes(w, h, seed) if kind == "bytes" else S.noise_frame(w, h, seed=seed), 1)[0]
    oxs, oys = O.detect(plane, *rect, margin, n, dist, quality)
    assert 4 < len(oxs) < n  # every candidate was looked at
    d = torch.from_numpy(plane).cuda()
    torch.cuda.synchronize()
    det = vtg_lib.Detector(ctx, w, h)
    for _ in range(4):
        xs, ys = det.detect(d.data_ptr(), w, h, w, *rect, margin, n, dist, quality)
        assert np.array_equal(xs, oxs) and np.array_equal(ys, oys)
    det.close()
