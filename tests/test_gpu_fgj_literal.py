"""The Jacobi foreground's own form (n - 1 iterations a level, resizes read on
the way, the first levels in one launch) against the buffer-by-buffer one that
calls with an iteration count of zero take: with every level small, the count
of the large ones does not enter, so both make the same result, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Up to 8192 pixels a level is one CTA's in the buffer-by-buffer form; 3400 is
# what the first levels' launch holds.
@pytest.mark.parametrize("h,w", [(1, 2), (2, 2), (17, 1), (1, 90), (58, 58), (59, 58), (68, 50), (65, 64), (90, 91),
                                 (91, 91), (40, 129), (257, 190)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 11])
def test_own_form_and_buffers(gpu, h, w, n):
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * 100 + w + n)
    img = rng.random((h, w, 3)).astype(np.float32)
    alpha = np.clip(rng.random((h, w)) * 1.4 - 0.2, 0.0, 1.0).astype(np.float32)
    alpha[rng.random((h, w)) < 0.3] = 0.0
    kw = dict(n_small_iterations=n, small_size=65535, return_background=True)
    own = pm.estimate_foreground_ml_cupy(img, alpha, n_big_iterations=1, **kw)
    buffers = pm.estimate_foreground_ml_cupy(img, alpha, n_big_iterations=0, **kw)
    for a, b in zip(own, buffers):
        assert np.array_equal(a, b)
