"""The still picture's cell differences once its mean is fractional (the third frame on): the F32 sums' order shows then, and is the
warp's, element k in partial sum k % 32 and the partial sums by a butterfly of strides 1, 2, 4, 8, 16. Compared bit for bit with
those sums formed here from the mean that the frame before left."""
import numpy as np
import pytest

import oracle as O
import vtg_synth as S

pytestmark = pytest.mark.gpu


def _diffs(mean, cur, cols, rows):
    h, w = cur.shape
    out = np.zeros(cols * rows, np.float32)
    for r in range(rows):
        y1 = min(8 * r + 8, h)
        for c in range(cols):
            xs = np.minimum(np.arange(16 * c, 16 * c + 16), w - 1)
            d = np.abs(cur[8 * r:y1, xs] - mean[8 * r:y1, xs]).astype(np.float32).ravel()
            part = np.zeros(32, np.float32)
            for k in range(0, len(d), 32):
                part[:len(d[k:k + 32])] += d[k:k + 32]
            for s in (1, 2, 4, 8, 16):
                part = part + part[np.arange(32) ^ s]
            out[r * cols + c] = part[0] / np.float32(len(d)) * np.float32(1 / 64)
    return out


@pytest.mark.parametrize("w,h", [(64, 48), (83, 61), (320, 200)])
@pytest.mark.parametrize("avg", [3, 16])
def test_differences_from_a_fractional_mean(vtg_lib, ctx, w, h, avg):
    import torch

    rng = np.random.default_rng(w)
    base = S.noise_frame(w, h, seed=w).astype(int)
    st = vtg_lib.Still(ctx, w, h, avg, 1.0, 40.0)
    mean, fractional = None, 0
    for k in range(7):
        cur = O.pyramid(np.clip(base + rng.integers(-3, 4, base.shape), 0, 255).astype(np.uint8), 1)[0]
        d = torch.from_numpy(cur).cuda()
        torch.cuda.synchronize()
        st.frame(d.data_ptr(), w)
        cells, motion, after = st.read()
        if k >= 3:
            fractional += bool((mean != np.round(mean)).any())  # not after four frames: multiples of 64 divided by four
            assert cells["diff"].tobytes() == _diffs(mean, cur, st.cols, st.rows).tobytes(), k
        mean = after
    assert fractional >= 2
    st.close()
