"""A template with values that FP16 does not hold, and a norm at which its scores still count: the F32 search of bytes leaves the FP16
filter out, and its map is the F32 plane's bit for bit. Large templates over most of the plane take their window sums from the
integral images then, on bytes too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spiked(frame, tw, th, spikes):
    """A cut template with a few values past 65,504, and a hundredth of its norm, so that windows of random bytes are not near-blank beside it."""
    patch = frame[8:8 + th, 5:5 + tw].astype(np.float32)
    app = (patch - np.float32(patch.mean(dtype=np.float64))).astype(np.float32)
    for k, v in enumerate(spikes):
        app[th // 2, tw // 3 + 5 * k] = v
    return app, float(np.sum(app.astype(np.float64) ** 2)) / 100


@pytest.mark.parametrize("spikes", [(7e4,), (-7e4,), (7e4, -7e4), (6.6e4, 3e4)])
@pytest.mark.parametrize("w,h,tw,th,step", [(300, 300, 72, 72, 1), (300, 300, 72, 72, 2), (330, 250, 64, 64, 1), (300, 200, 128, 40, 1),
                                            (620, 480, 32, 40, 1)])
def test_templates_past_fp16_take_the_direct_map(vtg_lib, ctx, w, h, tw, th, step, spikes):
    import torch

    frame = np.random.default_rng(w + h).integers(0, 256, (h, w)).astype(np.uint8)  # windows with contrast enough for such a norm
    app, norm = spiked(frame, tw, th, spikes)
    u8 = torch.from_numpy(frame).cuda()
    f32 = torch.from_numpy(frame.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = vtg_lib.Search(ctx, w, h)
    s.template(app, norm)
    a = s.run(u8.data_ptr(), w, h, w, vtg_lib.PLANE_U8, 1, w, 1, h, step, want_map=True)
    b = s.run(f32.data_ptr(), w, h, w, vtg_lib.PLANE_F32, 1, w, 1, h, step, want_map=True)
    s.close()
    assert (b[1] != 0).mean() > 0.9  # scores, not near-blank windows' zeros
    assert a[0] == b[0]
    for p, q in zip(a[1:], b[1:]):
        assert p.tobytes() == q.tobytes()
