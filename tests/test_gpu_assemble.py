"""The radius-1 assembly at the edges of its 32 x 8 tiles: bit-identical to
the oracle's Laplacian (itself pinned to the reference), with and without
known windows, on noise, flat and extreme images."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(1, 5), (2, 33), (3, 3), (7, 31), (8, 32), (9, 33), (10, 34), (17, 64),
                                 (16, 65), (25, 97)])
@pytest.mark.parametrize("kind", ["noise", "flat", "steps", "tiny"])
def test_radius1_bit_exact(gpu, h, w, kind):
    import pymatting_b200 as pm
    rng = np.random.default_rng(h * 100 + w)
    img = rng.random((h, w, 3))
    if kind == "flat":
        img[:] = 0.25
    elif kind == "steps":
        img = np.round(img * 3) / 3
    elif kind == "tiny":
        img *= 1e-160
    known = rng.random((h, w)) < 0.7
    for mask in (None, known):
        L = pm.cf_laplacian(img, is_known=mask)
        Lr = oracle.cf_laplacian(img, is_known=mask)
        assert np.array_equal(L.indptr, Lr.indptr) and np.array_equal(L.indices, Lr.indices)
        assert np.array_equal(L.data, Lr.data)
    tri = np.where(known, np.where(img[:, :, 0] > img.mean(), 1.0, 0.0), 0.5)
    tri[0, 0], tri[-1, -1] = 0.0, 1.0
    A, _b = pm.make_linear_system(pm.cf_laplacian(img), tri)
    Ar, _br = oracle.make_linear_system(oracle.cf_laplacian(img), tri)
    d = pm.jacobi(A)                   # the planes' diagonal
    assert np.array_equal(d(np.ones(h * w)), 1.0 / Ar.diagonal())


@pytest.mark.parametrize("h,w", [(9, 33), (16, 65)])
def test_planes_equal_rows(gpu, h, w):
    """The half-stencil planes hold the forward entries of the rows."""
    import pymatting_b200 as pm
    from pymatting_b200.laplacian import device_source
    rng = np.random.default_rng(3)
    A = pm.cf_laplacian(rng.random((h, w, 3)))
    src = device_source(A)
    planes = src.planes().cpu().numpy().reshape(13, h, -1)[:, :, :w]
    values = src.ell()[0].cpu().numpy().reshape(h, w, 5, 5)
    offsets = [(0, 0), (0, 1), (0, 2)] + [(dy, dx) for dy in (1, 2) for dx in range(-2, 3)]
    for p, (dy, dx) in enumerate(offsets):
        y, x = np.mgrid[:h, :w]
        inside = (y + dy < h) & (x + dx >= 0) & (x + dx < w)
        assert np.array_equal(planes[p], np.where(inside, values[:, :, dy + 2, dx + 2], 0.0))
