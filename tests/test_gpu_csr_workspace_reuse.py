"""A CSR system made while the memory that becomes its workspace is still
written to, and read, by work queued on the caller's stream."""

import numpy as np
import pytest
import scipy.sparse

pytestmark = pytest.mark.gpu


def _system(n, csr):
    from pymatting_b200.systems import M_NONE, CsrSystem
    return CsrSystem(n, M_NONE, csr=csr)


@pytest.mark.parametrize("n", [300, 40000])
def test_workspace_in_use_when_bound(gpu, n):
    import torch
    from pymatting_b200.solver import to_device_csr
    csr = to_device_csr(scipy.sparse.diags([-1.0, 2.5, -1.0], [-1, 0, 1], (n, n)).tocsr())[:3]
    b = torch.rand(n, dtype=torch.float64, device=gpu, generator=torch.Generator(gpu).manual_seed(1))
    first = _system(n, csr)
    assert first.stats().iters == 0 and first.stats().status == 0
    want, iters = first.solve(b).clone(), first.stats().iters
    nbytes = first.workspace.numel()
    for _ in range(3):
        torch.cuda.synchronize()
        block = torch.full((nbytes,), 7, dtype=torch.uint8, device=gpu)
        torch.cuda._sleep(20_000_000)
        total = block.sum(dtype=torch.int64)         # reads what a bind must not touch
        block.fill_(255)                             # writes what a solve must not see
        del block
        system = _system(n, csr)
        x = system.solve(b)
        assert torch.equal(x, want) and system.stats().iters == iters
        assert int(total) == 7 * nbytes
