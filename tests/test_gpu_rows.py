"""The row-streaming stencil kernels (CG apply, restriction, prolongation) at
the sizes where their strips and segments end: widths around multiples of 58,
60, 116 and 120 columns, heights from one row up, odd and even.

Tolerances: the FP64 V-cycle does at most 60 operations per pixel and level
on 8 levels, so its rounding stays below 8 * 60 * 1.1e-16 = 5e-14 of the
largest entry times the smoother's amplification (about 10): 1e-12. The
operator apply is one level: 1e-14 of sum |a| |x|. The mixed solve is held to
the 1e-4 that its alphas are promised for, at relative residual 1e-11."""

import numpy as np
import pytest

import oracle
from pymatting_b200.synthetic import make_matting_problem

pytestmark = pytest.mark.gpu

SIZES = [(2, 64), (3, 59), (9, 57), (8, 58), (7, 60), (10, 61), (33, 62), (12, 115), (31, 117),
         (17, 119), (5, 121), (66, 123), (130, 33), (257, 5), (64, 180), (35, 241)]


def _problem(h, w, seed):
    rng = np.random.default_rng(seed)
    img = rng.random((h, w, 3))
    tri = np.full((h, w), 0.5)
    tri[rng.random((h, w)) < 0.3] = 0.0
    tri[rng.random((h, w)) < 0.3] = 1.0
    tri[0, 0], tri[-1, -1] = 0.0, 1.0
    return img, tri


@pytest.mark.parametrize("h,w", [s for s in SIZES if s[0] >= 3])
def test_fp64_vcycle_and_apply(gpu, h, w):
    import torch
    import pymatting_b200 as pm
    img, tri = _problem(h, w, h * 1000 + w)
    A, _b = pm.make_linear_system(pm.cf_laplacian(img), tri)
    Ar, _br = oracle.make_linear_system(oracle.cf_laplacian(img), tri)
    v = np.random.default_rng(1).standard_normal(h * w)
    M = pm.vcycle(A, (h, w))
    z, zr = M(v), oracle.vcycle(Ar, (h, w))(v)
    assert np.abs(z - zr).max() <= 1e-12 * np.abs(zr).max()
    y = M.system.apply(torch.from_numpy(v).to(gpu)).cpu().numpy()
    scale = abs(Ar).dot(np.abs(v))
    assert (np.abs(y - Ar.dot(v)) <= 1e-14 * scale).all()


@pytest.mark.parametrize("vec", [2, 4])
def test_mixed_batch_of_edge_sizes(gpu, vec):
    from pymatting_b200 import autotune
    from pymatting_b200.batch import AlphaBatch
    sizes = [s for s in SIZES if min(s) >= 31]
    probs = [make_matting_problem(h, w, 7 + h + w, sigma=1.0, band=1, unknown_fraction=0.3)[:2]
             for h, w in sizes]
    batch = AlphaBatch([p[0] for p in probs], [p[1] for p in probs], precision="mixed")
    autotune.apply_tuning(batch.system, {"vec_apply": vec, "vec_up": vec})
    alphas = batch.alphas(batch.solve(rtol=1e-11))
    for a, (img, tri) in zip(alphas, probs):
        ref = np.clip(oracle.soft_alpha_exact(img, tri), 0, 1)
        assert np.abs(a.cpu().numpy() - ref.reshape(tri.shape)).max() <= 1e-4
