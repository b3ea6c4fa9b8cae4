"""The streamed triangular solves where a row's terms change hands: 64 of them
come through registers, the others in groups of four per lane (128), and chunks
of more than eight rows give a warp a second row. Nothing discarded, so rows of
the factor are as long as the band. Against the oracle as in test_gpu_ichol."""

import pytest

from test_gpu_ichol import check_factor, grid_laplacian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [31, 32, 33, 63, 64, 65, 66, 95, 97, 160, 191, 192, 193, 320, 321])
def test_long_rows(gpu, w):
    import pymatting_b200 as pm
    check_factor(pm, grid_laplacian(5, w, 1e-2, w), discard_threshold=0.0)


@pytest.mark.parametrize("h,w", [(400, 4), (90, 90)])
def test_chunks_of_many_rows(gpu, h, w):
    import pymatting_b200 as pm
    check_factor(pm, grid_laplacian(h, w, 1e-1, w), discard_threshold=0.05)
