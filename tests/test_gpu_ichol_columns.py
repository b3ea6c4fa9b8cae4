"""The pipelined incomplete-Cholesky kernel (csrc/ichol.cu) where its rules
change: bandwidths around its chunks of 32 offsets, its finisher counts and its
largest (then the global front), fewer columns than warps, columns of several
hundred entries, and values outside the range of its quotient. Against the
oracle as in test_gpu_ichol (structure exact, values 1e-12), and by exact
scaling: with the matrix times 4^k, the factor is 2^k times the same bits."""

import numpy as np
import pytest
import scipy.sparse

from test_gpu_ichol import check_factor, grid_laplacian

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pm():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import pymatting_b200
    return pymatting_b200


@pytest.mark.parametrize("h,w", [(5, 1), (1, 7), (3, 2), (40, 15), (40, 16), (9, 31), (9, 32), (9, 33),
                                 (6, 64), (5, 65), (5, 129), (4, 256), (4, 257), (3, 512), (3, 513), (3, 1024),
                                 (3, 1025)])
def test_column_kernel_bandwidths(pm, h, w):
    check_factor(pm, grid_laplacian(h, w, 1e-2, h + w))
    check_factor(pm, grid_laplacian(h, w, 1e-2, h * w), discard_threshold=0.0,
                 relative_discard_threshold=1e-3, diag_keep_discarded=False)


def test_diagonal_matrix(pm):
    check_factor(pm, scipy.sparse.csc_matrix(scipy.sparse.diags(np.arange(1.0, 40.0))))


@pytest.mark.parametrize("w", [140, 300])
def test_dense_columns(pm, w):
    """No entry discarded: up to w entries behind each of w nodes."""
    A = grid_laplacian(4 if w == 300 else 8, w, 1e-2, w)
    check_factor(pm, A, discard_threshold=0.0)


@pytest.mark.parametrize("k", [-420, 300])
def test_values_outside_the_quotient_range(pm, k):
    A = grid_laplacian(12, 30, 1e-2, 5)
    L, r, p = pm.ichol(A, shifts=[0.0]).Ltuple
    B = scipy.sparse.csc_matrix(A)
    B.data = np.ldexp(B.data, 2 * k)
    Ls, rs, ps = pm.ichol(B, discard_threshold=float(np.ldexp(1e-4, k)), shifts=[0.0]).Ltuple
    np.testing.assert_array_equal(p, ps)
    np.testing.assert_array_equal(r, rs)
    np.testing.assert_array_equal(np.ldexp(L, k), Ls)
