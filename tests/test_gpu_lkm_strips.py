"""The fused box filters of the large-kernel Laplacian's apply (csrc/lkm.cu) at
the edges of its strips and row segments, at the smallest image of a radius,
and on both sides of its largest radius, against windows summed one by one in
float64. epsilon = 1e-3 keeps the windows' covariances at a condition of about
1e3 on noise, so rounding stays below (2r + 1)^2 1e3 2^-53 of the largest
value: 1e-9 for the radii here."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def direct(image, p, r, eps):
    h, w = p.shape
    n = (2 * r + 1) ** 2
    win = np.lib.stride_tricks.sliding_window_view
    I = win(image, (2 * r + 1, 2 * r + 1), axis=(0, 1)).reshape(h - 2 * r, w - 2 * r, 3, n)
    P = win(p, (2 * r + 1, 2 * r + 1)).reshape(h - 2 * r, w - 2 * r, n)
    d = I - I.mean(-1, keepdims=True)
    V = np.linalg.inv(d @ d.swapaxes(-1, -2) / n + eps / n * np.eye(3))
    dp = P - P.mean(-1, keepdims=True)
    g = V @ (d @ dp[..., None])[..., 0, None] / n              # (.., 3, 1)
    res = dp - (d * g).sum(-2)                                 # window residuals
    out = np.zeros((h, w))
    k = 0
    for dy in range(2 * r + 1):
        for dx in range(2 * r + 1):
            out[dy:dy + h - 2 * r, dx:dx + w - 2 * r] += res[..., k]
            k += 1
    return out


@pytest.mark.parametrize("h,w,r", [(3, 3, 1), (7, 128, 1), (9, 254, 1), (21, 21, 10), (22, 129, 10),
                                   (30, 236, 10), (41, 130, 5), (64, 33, 3), (66, 68, 32), (68, 67, 33)])
def test_lkm_apply_strips(h, w, r):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * w + r)
    image, p = rng.random((h, w, 3)), rng.standard_normal((h, w))
    ref = direct(image, p, r, 1e-3)
    L = pm.lkm_laplacian(image, epsilon=1e-3, radius=r, return_diagonal=False)
    np.testing.assert_allclose(np.asarray(L(p.ravel())).reshape(h, w), ref, rtol=0,
                               atol=1e-9 * np.abs(ref).max())
