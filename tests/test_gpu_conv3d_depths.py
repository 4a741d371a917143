"""Depths of the one-pass 3x3x3 convolution (sint_nn3d.cu) around its blocks of
output slices: 12 per thread up to 4 output channels, 8 up to 8, 4 up to 16.
49 x 70 nodes are 3 x 5 tiles, so every instance runs first, inner and partial
last slice blocks on tiles at the window's border and inside it (needs a B200).
"""
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


@pytest.mark.parametrize("cout,D", [(c, d) for c in (1, 2, 3) for d in (12, 13, 25, 37)] +
                         [(5, 8), (5, 9), (5, 25), (16, 4), (16, 9), (17, 1), (17, 3)])
def test_conv3d_depths(cout, D):
    from hpsint_b200 import predictor as P
    S, H, W, c1, c2 = 2, 49, 70, 2, 1
    rng = np.random.default_rng(100 * cout + D)
    f32 = lambda *shape: rng.normal(size=shape).astype(np.float32).astype(np.float64)
    x1, x2, w1, w2, b = f32(S, D, c1, H, W), f32(S, D, c2, H, W), f32(3, cout, c1, 3, 3), f32(3, cout, c2, 3, 3), f32(cout)
    dev = lambda a: torch.tensor(a, dtype=torch.float32, device="cuda")
    want = R.conv3x3x3(x1, w1, b) + R.conv3x3x3(x2, w2)
    # each partial sum of the 27 (c1 + c2) + 1 terms rounds by 2^-24 of at most the sum of magnitudes
    mag = R.conv3x3x3(abs(x1), abs(w1), abs(b)) + R.conv3x3x3(abs(x2), abs(w2))
    bound = (27 * (c1 + c2) + 2) * 2.0**-24 * mag
    out = torch.full((S, D + 2, cout, H, W), 7.0, device="cuda")
    P.conv3d_fused(padded(x1), dev(w1), out, x2=padded(x2), w2=dev(w2), bias=dev(b), slope=0.5)
    got = out.cpu().numpy().astype(np.float64)
    assert (got[:, 0] == 0).all() and (got[:, -1] == 0).all()
    assert (np.abs(got[:, 1:-1] - np.where(want < 0, 0.5 * want, want)) <= bound).all()
