"""Which kernel makes an incomplete Cholesky factor, and what follows when a
wait of the pipelined one runs out: the factor of the global front, identical."""

import numpy as np
import pytest

from pymatting_b200.preconditioner import CholeskyDecomposition, _csc_arrays
from test_gpu_ichol import check_factor, grid_laplacian

pytestmark = pytest.mark.gpu


def _factor(A, polls=-1, **kw):
    from pymatting_b200 import _ffi
    from pymatting_b200.systems import IcholFactor, csc_profile
    csc, n = _csc_arrays(A)
    band, envelope = csc_profile(csc, n)
    f = IcholFactor(n, band, max(envelope, n))
    assert f.kernel() is None
    _ffi.check(_ffi.lib().pmb_ichol_wait_limit(f._h, polls), "pmb_ichol_wait_limit")
    args = dict(discard=1e-4, shift=0.0, max_nnz=1 << 30, rel=0.0, keep=True)
    args.update(kw)
    nnz = f.factor(csc, args["discard"], args["shift"], args["max_nnz"], args["rel"], args["keep"])
    return f, nnz


@pytest.mark.parametrize("w", [1, 30, 300, 500, 1024])
def test_pipeline_bandwidths(gpu, w):
    f, nnz = _factor(grid_laplacian(4, w, 1e-2, w))
    assert nnz > 0 and f.kernel() == "pipeline"


def test_wider_bands_take_the_global_front(gpu):
    f, nnz = _factor(grid_laplacian(3, 1025, 1e-2, 1))
    assert nnz > 0 and f.kernel() == "global"


# 0 polls end every wait at once, a few let some columns through.
@pytest.mark.parametrize("polls", [0, 1, 3])
@pytest.mark.parametrize("h,w", [(20, 1), (12, 40), (8, 270), (6, 500)])
def test_a_wait_that_runs_out(gpu, h, w, polls):
    A = grid_laplacian(h, w, 1e-2, h * w)
    f, nnz = _factor(A, polls)
    if polls == 0:
        assert f.kernel() == "global after a pipeline wait ran out"
    g, mnz = _factor(A)
    assert g.kernel() == "pipeline" and nnz == mnz
    for a, b in zip(CholeskyDecomposition(f).Ltuple, CholeskyDecomposition(g).Ltuple):
        np.testing.assert_array_equal(a, b)
    assert f.levels() == g.levels()


def test_failure_codes_after_a_wait_that_ran_out(gpu):
    A = grid_laplacian(6, 30, 1e-2, 1)
    for polls in (-1, 0):
        assert _factor(A, polls, shift=-50.0)[1] == -1
        assert _factor(A, polls, discard=0.0, max_nnz=A.shape[0] + 10)[1] == -2
        f, nnz = _factor(A, polls)
        assert nnz > 0


# Bands around the first width with a cluster of 4 and the last that fits 8
# CTAs, nothing discarded: columns of nearly the whole band.
@pytest.mark.parametrize("w,kernel", [(250, "pipeline"), (290, "cluster"), (300, "cluster"), (400, "cluster"),
                                      (430, "cluster"), (446, "pipeline")])
@pytest.mark.parametrize("keep", [True, False])
def test_long_columns(gpu, w, kernel, keep):
    import pymatting_b200 as pm
    A = grid_laplacian(8, w, 1e-2, w)
    f, _nnz = _factor(A, discard=0.0, keep=keep)
    assert f.kernel() == kernel
    check_factor(pm, A, discard_threshold=0.0, diag_keep_discarded=keep)


def test_long_columns_are_seen_by_the_pipeline(gpu):
    """A small threshold: the pipeline's first columns tell, where there are
    many more to come. The factors are the same."""
    import pymatting_b200 as pm
    w = 400
    A = grid_laplacian(34, w, 1e-2, 3)
    assert _factor(A, discard=1e-14)[0].kernel() == "cluster"
    assert _factor(A, discard=1e-2)[0].kernel() == "pipeline"
    assert _factor(grid_laplacian(15, w, 1e-2, 3), discard=1e-14)[0].kernel() == "pipeline"
    check_factor(pm, A, discard_threshold=1e-14)


def test_failure_codes_of_long_columns(gpu):
    A = grid_laplacian(8, 300, 1e-2, 1)
    assert _factor(A, discard=0.0)[0].kernel() == "cluster"
    assert _factor(A, discard=0.0, shift=-50.0)[1] == -1
    assert _factor(A, discard=0.0, max_nnz=3 * A.shape[0])[1] == -2
