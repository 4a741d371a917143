"""Tilings of the one-pass 3x3x3 convolution of the 3D guess (sint_nn3d.cu): the
tile width is chosen for the window, with idle threads in tiles of fewer than
256 nodes."""
import numpy as np
import pytest
from oracle import predictor_ref as R

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def padded(a):
    """[S][D][C][H][W] with a zero slice below and above, FP32 on the device."""
    t = torch.zeros((a.shape[0], a.shape[1] + 2) + a.shape[2:], device="cuda")
    t[:, 1:-1] = torch.tensor(a, dtype=torch.float32)
    return t


# windows just below, at and above the edges of 16 x 16 and 32 x 8 tiles, and
# widths in between (25 x 25: tiles of 28 x 9, 49 x 70: 25 x 10)
@pytest.mark.parametrize("H,W", [(15, 15), (16, 16), (17, 48), (16, 33), (31, 15), (33, 33), (8, 32), (1, 1), (25, 25),
                                 (49, 70), (5, 97)])
@pytest.mark.parametrize("cout", [1, 2, 3, 5, 16, 17])
def test_conv3d_tilings(H, W, cout):
    from hpsint_b200 import predictor as P
    S, D, c1, c2, group = 2, 5, 3, 2, 2
    rng = np.random.default_rng(1000 * H + 10 * W + cout)
    f32 = lambda *shape: rng.normal(size=shape).astype(np.float32).astype(np.float64)
    x1, x2 = f32(S, D, c1, H, W), f32(S, D, c2, H, W)
    w1, w2, b = f32(3, cout, c1, 3, 3), f32(3, cout, c2, 3, 3), f32(cout)
    add, prev = f32(S // group, D, cout, H, W), f32(S, D, cout, H, W)
    dev = lambda a: torch.tensor(a, dtype=torch.float32, device="cuda")
    want = R.conv3x3x3(x1, w1, b) + R.conv3x3x3(x2, w2) + np.repeat(add, group, axis=0) + prev
    # FP32 sums of 27 (c1 + c2) + 3 terms: each partial sum rounds by 2^-24 of at
    # most the sum of magnitudes
    mag = (R.conv3x3x3(abs(x1), abs(w1), abs(b)) + R.conv3x3x3(abs(x2), abs(w2)) + np.repeat(abs(add), group, axis=0) +
           abs(prev))
    bound = (27 * (c1 + c2) + 4) * 2.0**-24 * mag
    out = padded(prev)
    out[:, 0], out[:, -1] = 7.0, -3.0
    P.conv3d_fused(padded(x1), dev(w1), out, x2=padded(x2), w2=dev(w2), bias=dev(b), addend=padded(add),
                   addend_group=group, slope=0.5, accumulate=True)
    got = out.cpu().numpy().astype(np.float64)
    assert (got[:, 0] == 0).all() and (got[:, -1] == 0).all()
    assert (np.abs(got[:, 1:-1] - np.where(want < 0, 0.5 * want, want)) <= bound).all()
