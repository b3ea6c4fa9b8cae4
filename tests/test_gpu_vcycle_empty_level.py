"""The V-cycle on long narrow images, whose levels halve to a grid without
pixels (300x3, 150x1, 75x0) before they are small enough to be solved
directly: like the reference, which then corrects by nothing there.

Tolerance: as in test_gpu_rows, at most 60 operations per pixel, level and
sweep on 8 levels with up to 4 sweeps, amplified by the smoother about 10
times: 4 * 60 * 8 * 1.1e-16 * 10 = 2e-12 of the largest entry."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# 64-bit tails hold levels of up to (16 * h * 32 * 8 bytes <= 227 KB): (1, 150)
# and (56, 0) are in one, (75, 0) is not.
SHAPES = [(300, 3), (3, 300), (226, 3), (3, 140), (3000, 40), (40, 3000), (700, 5)]


@pytest.mark.parametrize("h,w", SHAPES)
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2), (1, 2), (1, 0), (0, 1)])
def test_vcycle(gpu, h, w, pre, post):
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * 1000 + w)
    img, tri = rng.random((h, w, 3)), np.full((h, w), 0.5)
    tri[rng.random((h, w)) < 0.3] = 0.0
    tri[rng.random((h, w)) < 0.3] = 1.0
    A, _b = pm.make_linear_system(pm.cf_laplacian(img), tri)
    Ar, _br = oracle.make_linear_system(oracle.cf_laplacian(img), tri)
    v = rng.standard_normal(h * w)
    kw = dict(num_pre_iter=pre, num_post_iter=post)
    z, zr = pm.vcycle(A, (h, w), **kw)(v), oracle.vcycle(Ar, (h, w), **kw)(v)
    assert np.isfinite(zr).all()
    assert np.abs(z - zr).max() <= 2e-12 * np.abs(zr).max()


def test_mixed_batch_with_an_empty_level(gpu):
    from pymatting_b200.batch import AlphaBatch
    from pymatting_b200.synthetic import make_matting_problem
    probs = [make_matting_problem(h, w, h + w, sigma=1.0, band=1, unknown_fraction=0.3)[:2]
             for h, w in [(300, 3), (33, 47), (3, 300), (64, 64)]]
    batch = AlphaBatch([p[0] for p in probs], [p[1] for p in probs], precision="mixed")
    for a, (img, tri) in zip(batch.alphas(batch.solve(rtol=1e-11)), probs):
        ref = np.clip(oracle.soft_alpha_exact(img, tri), 0, 1)
        assert np.abs(a.cpu().numpy() - ref.reshape(tri.shape)).max() <= 1e-4
