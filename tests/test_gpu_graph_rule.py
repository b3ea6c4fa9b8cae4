"""First solves that go on by a graph after their first iterations: the same
kernels on the same data as later solves, which replay it from the start, so
the same bits and the same number of iterations. Iteration counts on both sides
of the lines (36 for CSR systems, 96 and 192 for stencil systems)."""

import numpy as np
import pytest

from pymatting_b200.synthetic import make_matting_problem

pytestmark = pytest.mark.gpu


def _stencil(precision, preconditioner):
    import torch
    import pymatting_b200 as pm
    from pymatting_b200.laplacian import device_source
    from pymatting_b200.systems import StencilSystem
    img, tri = make_matting_problem(24, 32, 3, sigma=2.0, band=3, unknown_fraction=0.25)[:2]
    A, b = pm.make_linear_system(pm.cf_laplacian(img), tri)
    system = StencilSystem([device_source(A)], precision, preconditioner)
    system.setup()
    return system, torch.from_numpy(np.asarray(b)).cuda()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("preconditioner", [0, 1, 2])
@pytest.mark.parametrize("maxiter", [1, 95, 96, 97, 101, 191, 192, 193, 230])
def test_stencil_first_solve(gpu, precision, preconditioner, maxiter):
    import torch
    system, b = _stencil(precision, preconditioner)
    runs = []
    for _ in range(3):
        x = system.solve(b, None, 0.0, 1e-9, maxiter, False)
        st = system.stats(0)
        runs.append((x.clone(), st.iters, st.status, st.norm_r))
    assert all(r[1:] == runs[0][1:] and torch.equal(r[0], runs[0][0]) for r in runs)
    assert runs[0][1] <= maxiter


@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("maxiter", [1, 35, 36, 37, 41, 90])
def test_csr_first_solve(gpu, jacobi, maxiter):
    import torch
    import scipy.sparse
    from pymatting_b200.solver import to_device_csr
    from pymatting_b200.systems import M_JACOBI, M_NONE, CsrSystem
    n = 700
    A = scipy.sparse.diags([-1.0, 2.01, -1.0], [-1, 0, 1], (n, n)).tocsr()
    indptr, indices, data, _n, _m = to_device_csr(A)
    b = torch.rand(n, dtype=torch.float64, device=gpu, generator=torch.Generator(gpu).manual_seed(1))
    inv = torch.full((n,), 1 / 2.01, dtype=torch.float64, device=gpu) if jacobi else None
    system = CsrSystem(n, M_JACOBI if jacobi else M_NONE, csr=(indptr, indices, data), inv_diag=inv)
    runs = []
    for _ in range(3):
        x = system.solve(b, None, 0.0, 1e-12, maxiter, False)
        st = system.stats()
        runs.append((x.clone(), st.iters, st.status, st.norm_r))
    assert all(r[1:] == runs[0][1:] and torch.equal(r[0], runs[0][0]) for r in runs)
    assert runs[0][1] <= maxiter
