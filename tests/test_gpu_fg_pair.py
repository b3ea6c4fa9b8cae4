"""The foreground sweeps at the sizes where their kernels change or end:
levels up to 32x32 and beyond, strips of 32 rows that end full, with one row
or in the middle, widths below and around a chunk of 8 steps, one, two and
three iterations. Bit-identical to the oracle for its seed colours."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(32, 32), (33, 3), (33, 32), (32, 33), (64, 9), (65, 40), (96, 41), (97, 100),
                                 (31, 150), (3, 210)])
@pytest.mark.parametrize("n_big", [1, 2, 3])
def test_sweeps_bit_exact(gpu, h, w, n_big):
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * 1000 + w)
    depth = 1 + (h + w) % 4
    img = rng.random((h, w, depth)).astype(np.float32)
    alpha = np.clip(rng.random((h, w)) * 1.4 - 0.2, 0.0, 1.0).astype(np.float32)
    seed = oracle.fg_mean_colors(img, alpha)
    F, B = pm.estimate_foreground_ml(img, alpha, return_background=True, seed_colors=seed,
                                     n_big_iterations=n_big)
    Fr, Br = oracle.estimate_foreground_ml(img, alpha, return_background=True, n_big_iterations=n_big)
    assert np.array_equal(F, Fr) and np.array_equal(B, Br)


def test_values_beyond_one(gpu):
    """Image values above 1 (starting colours that a clamped pair cannot be)."""
    import pymatting_b200 as pm
    rng = np.random.default_rng(5)
    img = (rng.random((70, 75, 3)) * 5 - 1).astype(np.float32)
    alpha = rng.random((70, 75)).astype(np.float32)
    seed = oracle.fg_mean_colors(img, alpha)
    for n_big in (1, 2):
        F, B = pm.estimate_foreground_ml(img, alpha, return_background=True, seed_colors=seed,
                                         n_big_iterations=n_big)
        Fr, Br = oracle.estimate_foreground_ml(img, alpha, return_background=True, n_big_iterations=n_big)
        assert np.array_equal(F, Fr) and np.array_equal(B, Br)
