"""The row-streaming kernels with their rows cut into other segments (the
autotuner's CTAs per SM): a pixel's value does not depend on the cut, and the
mixed solve, whose dot products do, keeps the accuracy that it promises (as in
test_gpu_rows)."""

import numpy as np
import pytest

import oracle
from pymatting_b200.synthetic import make_matting_problem
from test_gpu_rows import SIZES, _problem

pytestmark = pytest.mark.gpu

CUTS = [dict(ctas_fine=1, ctas_up=1, ctas_down=1), dict(ctas_fine=4, ctas_up=4, ctas_down=4),
        dict(ctas_fine=2, ctas_up=1, ctas_down=4)]


@pytest.mark.parametrize("h,w", [s for s in SIZES if s[0] >= 9] + [(300, 411)])
def test_vcycle_and_apply_are_the_same(gpu, h, w):
    import torch
    import pymatting_b200 as pm
    from pymatting_b200 import autotune
    img, tri = _problem(h, w, h + w)
    A, _b = pm.make_linear_system(pm.cf_laplacian(img), tri)
    M = pm.vcycle(A, (h, w))
    v = torch.from_numpy(np.random.default_rng(1).standard_normal(h * w)).to(gpu)
    z, y = M(v).clone(), M.system.apply(v).clone()
    for cut in CUTS:
        autotune.apply_tuning(M.system, cut)
        assert torch.equal(M(v), z) and torch.equal(M.system.apply(v), y)


@pytest.mark.parametrize("cut", CUTS)
def test_mixed_batch(gpu, cut):
    from pymatting_b200 import autotune
    from pymatting_b200.batch import AlphaBatch
    probs = [make_matting_problem(h, w, 7 + h + w, sigma=1.0, band=1, unknown_fraction=0.3)[:2]
             for h, w in SIZES if min(h, w) >= 31]
    batch = AlphaBatch([p[0] for p in probs], [p[1] for p in probs], precision="mixed")
    autotune.apply_tuning(batch.system, cut)
    for a, (img, tri) in zip(batch.alphas(batch.solve(rtol=1e-11)), probs):
        ref = np.clip(oracle.soft_alpha_exact(img, tri), 0, 1)
        assert np.abs(a.cpu().numpy() - ref.reshape(tri.shape)).max() <= 1e-4
