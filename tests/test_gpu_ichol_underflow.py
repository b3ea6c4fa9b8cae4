"""Entries whose quotient underflows to -0.0, with a negative threshold that
keeps everything: they count, so they must have their place in the factor."""

import numpy as np
import pytest
import scipy.sparse

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,band", [(2, 1), (40, 1), (60, 9), (90, 40)])
def test_underflow_is_kept(gpu, n, band):
    import pymatting_b200 as pm
    rng = np.random.default_rng(n)
    diagonals, offsets = [np.full(n, 4.0)], [0]
    for o in sorted({1, band}):
        v = np.where(rng.random(n - o) < 0.5, -5e-324, -0.1)
        v[0] = -5e-324
        diagonals += [v, v]
        offsets += [o, -o]
    A = scipy.sparse.csc_matrix(scipy.sparse.diags(diagonals, offsets))
    kw = dict(discard_threshold=-1.0, shifts=[0.0])
    L, r, p = pm.ichol(A, **kw).Ltuple
    Lr, rr, pr = oracle.ichol(A, **kw).Ltuple
    assert (Lr[1:2] == 0.0).all() and np.signbit(Lr[1])
    np.testing.assert_array_equal(p, pr)
    np.testing.assert_array_equal(r, rr)
    np.testing.assert_allclose(L, Lr, rtol=1e-12, atol=0.0)
