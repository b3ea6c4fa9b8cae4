"""knn_laplacian at the edges of its tiles (32 points), windows (1024) and row
sorters (256 and 1024 entries): identical to the oracle, which keeps the k
smallest by (distance, index) like the kernel."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _same(L, Lr):
    # scipy's subtraction I - W drops entries that cancel (k = 1: all of them);
    # the device matrix stores them.
    L, Lr = L.tocsr().copy(), Lr.tocsr()
    L.eliminate_zeros()
    Lr.eliminate_zeros()
    Lr.sort_indices()
    assert np.array_equal(L.indptr, Lr.indptr) and np.array_equal(L.indices, Lr.indices)
    assert np.array_equal(L.data, Lr.data)


@pytest.mark.parametrize("h,w,ks", [(1, 31, [5]), (4, 8, [32, 3]), (3, 11, [20, 10]), (5, 13, [64]),
                                    (31, 33, [20, 10]), (32, 32, [1]), (41, 25, [7, 20])])
@pytest.mark.parametrize("kernel", ["binary", "soft"])
def test_sizes(gpu, h, w, ks, kernel):
    import pymatting_b200 as pm
    img = np.random.default_rng(h * w).random((h, w, 3))
    dws = [2.0, 0.1][:len(ks)]
    kw = dict(n_neighbors=ks, distance_weights=dws, kernel=kernel)
    _same(pm.knn_laplacian(img, **kw), oracle.knn_laplacian(img, **kw))


@pytest.mark.parametrize("h,w", [(10, 26), (25, 24), (30, 50)])
def test_equal_points(gpu, h, w):
    """All points equal: every row lists the first k, whose rows hold n entries.
    (Off the diagonal: a row that does not list itself has no stored diagonal
    on the device.)"""
    import pymatting_b200 as pm
    img = np.full((h, w, 3), 0.5)
    kw = dict(n_neighbors=[6], distance_weights=[0.0])
    L, Lr = pm.knn_laplacian(img, **kw).toarray(), oracle.knn_laplacian(img, **kw).toarray()
    off = ~np.eye(h * w, dtype=bool)
    assert np.array_equal(L[off], Lr[off])


def test_ties_and_clusters(gpu):
    """Few distinct colours on a grid: distances tie in every list."""
    import pymatting_b200 as pm
    rng = np.random.default_rng(2)
    img = rng.integers(0, 3, (40, 60, 3)) / 2.0
    _same(pm.knn_laplacian(img), oracle.knn_laplacian(img))
