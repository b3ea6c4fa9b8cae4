"""The Jacobi foreground at the edges of its 32 x 8 tiles and of the levels
that one CTA holds (3400 pixels), for one to three iterations, against the
oracle's restatement with the elementwise tolerance of the other Jacobi tests
(float32 rounding, amplified in near-singular pixels of the first levels)."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(58, 58), (59, 58), (68, 50), (8, 33), (65, 64), (63, 97), (40, 129)])
@pytest.mark.parametrize("n_small,n_big", [(10, 2), (1, 1), (3, 3), (10, 1)])
def test_jacobi_edges(gpu, h, w, n_small, n_big):
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * 100 + w)
    img = rng.random((h, w, 3)).astype(np.float32)
    alpha = np.clip(rng.random((h, w)) * 1.4 - 0.2, 0.0, 1.0).astype(np.float32)
    kw = dict(n_small_iterations=n_small, n_big_iterations=n_big, return_background=True)
    F, B = pm.estimate_foreground_ml_cupy(img, alpha, **kw)
    Fr, Br = oracle.estimate_foreground_ml_cupy(img, alpha, **kw)
    for x, r in ((F, Fr), (B, Br)):
        assert np.abs(x - r).max() <= 1e-3
    F1 = pm.estimate_foreground_ml_cupy(img, alpha, n_small_iterations=n_small, n_big_iterations=n_big)
    assert np.array_equal(F, F1)
