"""knn_laplacian on images with pixels that are not finite. Their rows mean
little, but the matrix must stay one: nothing here multiplies with it."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _bad_image(h, w, seed, bad, flat=False):
    rng = np.random.default_rng(seed)
    img = np.full((h, w, 3), 0.5) if flat else rng.random((h, w, 3))
    for k, v in enumerate(bad):
        img.reshape(-1, 3)[(h * w // 2 + 7 * k) % (h * w), k % 3] = v
    return img


# Equal points with distance weight 0 all list the same ones, whose rows then
# hold up to 256 entries (sorted by a warp), up to 1024 (a CTA), more (a thread).
@pytest.mark.parametrize("h,w,ks,flat", [(6, 9, [20, 10], False), (24, 25, [20, 10], False),
                                         (10, 10, [6, 4], True), (15, 20, [6, 4], True), (25, 28, [6, 4], True)])
@pytest.mark.parametrize("bad", [[np.nan], [np.inf], [np.nan, np.inf, -np.inf]])
@pytest.mark.parametrize("kernel", ["binary", "soft"])
def test_pattern(gpu, h, w, ks, flat, bad, kernel):
    import pymatting_b200 as pm
    n = h * w
    img = _bad_image(h, w, n, bad, flat)
    L = pm.knn_laplacian(img, n_neighbors=ks, distance_weights=[0.0, 0.0] if flat else [2.0, 0.1], kernel=kernel)
    indptr, indices, data = L.indptr, L.indices, L.data
    assert indptr[0] == 0 and indptr[-1] == len(indices) == len(data)
    assert (np.diff(indptr) >= ks[0]).all()
    assert indices.min() >= 0 and indices.max() < n
    row = np.repeat(np.arange(n), np.diff(indptr))
    assert (np.diff(row * n + indices) > 0).all()      # ascending and distinct in every row
    if kernel == "binary":
        assert np.isfinite(data).all()


def _knn_nan_last(f, k):
    """The k smallest by (distance, index), a NaN distance as infinite."""
    d = np.zeros((len(f), len(f)))
    for c in range(f.shape[1]):
        e = f[:, None, c] - f[None, :, c]
        d += (e * e).astype(np.float64)
    d[np.isnan(d)] = np.inf
    idx = np.broadcast_to(np.arange(len(f)), d.shape)
    return np.lexsort((idx, d), axis=1)[:, :k]


@pytest.mark.parametrize("at", [100, 117, 333, 590])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("kernel", ["binary", "soft"])
def test_one_bad_pixel_leaves_the_others_alone(gpu, monkeypatch, at, bad, kernel):
    """Only the pixel's own list is arbitrary: the k first pixels. Values are
    compared in the rows whose weights are finite, columns in all rows."""
    import pymatting_b200 as pm
    lists = []

    def knn(f, k):
        lists.append(_knn_nan_last(f, k))
        return lists[-1]

    monkeypatch.setattr(oracle, "knn", knn)
    h, w = 20, 30
    n = h * w
    img = np.random.default_rng(1).random((h, w, 3))
    img.reshape(-1, 3)[at, 1] = bad
    kw = dict(n_neighbors=[7], distance_weights=[1.0], kernel=kernel)
    with np.errstate(all="ignore"):
        Lr = oracle.knn_laplacian(img, **kw).toarray()
        L = pm.knn_laplacian(img, **kw)
        dense = L.toarray()
    pattern = np.zeros((n, n), bool)
    pattern[np.repeat(np.arange(n), 7), lists[0].ravel()] = True
    pattern |= pattern.T
    stored = np.zeros((n, n), bool)
    stored[np.repeat(np.arange(n), np.diff(L.indptr)), L.indices] = True
    # The pixel does not list itself, so its own diagonal is left out here.
    pattern[at, at] = stored[at, at] = False
    dense[at, at] = Lr[at, at] = 0.0
    assert np.array_equal(stored, pattern)
    fine = ~pattern[:, at]
    fine[at] = False
    fine |= kernel == "binary"
    assert np.array_equal(dense[fine], Lr[fine])


@pytest.mark.parametrize("n_bad", [31, 33, 100, 600])
def test_tiles_of_bad_pixels(gpu, monkeypatch, n_bad):
    """Whole tiles of 32 points without a finite one; the last has 24 points."""
    import pymatting_b200 as pm
    monkeypatch.setattr(oracle, "knn", _knn_nan_last)
    img = np.random.default_rng(2).random((20, 30, 3))
    img.reshape(-1, 3)[np.random.default_rng(3).permutation(600)[:n_bad]] = np.nan
    kw = dict(n_neighbors=[7, 5], distance_weights=[1.0, 0.1])
    with np.errstate(all="ignore"):
        Lr = oracle.knn_laplacian(img, **kw).toarray()
    assert np.array_equal(pm.knn_laplacian(img, **kw).toarray(), Lr)
