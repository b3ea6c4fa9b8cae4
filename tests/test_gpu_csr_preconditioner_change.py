"""A CSR system whose preconditioner is set anew between solves takes the new
one, also where earlier solves left a graph of iterations."""

import numpy as np
import pytest
import scipy.sparse

pytestmark = pytest.mark.gpu


def _csr(A):
    from pymatting_b200.solver import to_device_csr
    return to_device_csr(scipy.sparse.csr_matrix(A))[:3]


def test_matrix(gpu):
    import torch
    from pymatting_b200 import _ffi, _device as dev
    from pymatting_b200.systems import M_MATRIX, CsrSystem
    n = 500
    A = scipy.sparse.diags([-1.0, 2.5, -1.0], [-1, 0, 1], (n, n))
    d = np.random.default_rng(1).uniform(0.5, 2.0, n)
    m1, m2 = _csr(scipy.sparse.identity(n)), _csr(scipy.sparse.diags(d))
    b = torch.rand(n, dtype=torch.float64, device=gpu, generator=torch.Generator(gpu).manual_seed(1))
    fresh = CsrSystem(n, M_MATRIX, csr=_csr(A), m_csr=m2)
    want = fresh.solve(b).clone()
    system = CsrSystem(n, M_MATRIX, csr=_csr(A), m_csr=m1)
    for _ in range(2):
        system.solve(b)
    _ffi.check(_ffi.lib().pmb_csr_set_matrix_preconditioner(
        system._h, 0, dev.ptr(m2[0]), dev.ptr(m2[1]), dev.ptr(m2[2]), dev.stream()), "set")
    assert torch.equal(system.solve(b), want)
    assert system.stats().iters == fresh.stats().iters


def test_factor(gpu):
    import torch
    import pymatting_b200 as pm
    from pymatting_b200 import _ffi, _device as dev
    from pymatting_b200.systems import M_ICHOL, CsrSystem
    n = 500
    A = scipy.sparse.csc_matrix(scipy.sparse.diags([-1.0, -1.0, 5.0, -1.0, -1.0], [-20, -1, 0, 1, 20], (n, n)))
    f1, f2 = pm.ichol(A, discard_threshold=0.5).factor, pm.ichol(A, discard_threshold=1e-3).factor
    b = torch.rand(n, dtype=torch.float64, device=gpu, generator=torch.Generator(gpu).manual_seed(1))
    fresh = CsrSystem(n, M_ICHOL, csr=_csr(A), ichol=f2)
    want = fresh.solve(b).clone()
    system = CsrSystem(n, M_ICHOL, csr=_csr(A), ichol=f1)
    for _ in range(2):
        system.solve(b)
    assert system.stats().iters > fresh.stats().iters
    _ffi.check(_ffi.lib().pmb_csr_set_ichol(system._h, f2._h, dev.stream()), "set")
    assert torch.equal(system.solve(b), want)
    assert system.stats().iters == fresh.stats().iters
