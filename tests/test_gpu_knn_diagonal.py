"""knn_laplacian where pixels do not list themselves: more than k equal points
before them. The whole matrix against the oracle, diagonal included."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


# Rows of 256 entries and one more (a warp sorts them, a CTA), 1024 and more.
@pytest.mark.parametrize("h,w", [(2, 5), (10, 25), (25, 10), (7, 36), (30, 34), (31, 35)])
@pytest.mark.parametrize("kw", [dict(n_neighbors=[6], distance_weights=[0.0]),
                                dict(n_neighbors=[4, 3], distance_weights=[0.0, 0.0], kernel="soft"),
                                dict(n_neighbors=[1, 5], distance_weights=[0.0, 2.0])])
def test_equal_points_whole_matrix(gpu, h, w, kw):
    import pymatting_b200 as pm
    img = np.full((h, w, 3), 0.5)
    L, Lr = pm.knn_laplacian(img, **kw), oracle.knn_laplacian(img, **kw)
    assert np.array_equal(L.toarray(), Lr.toarray())
    assert (np.diff(L.indices) > 0)[np.diff(np.repeat(np.arange(h * w), np.diff(L.indptr))) == 0].all()
