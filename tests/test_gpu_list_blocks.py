"""Lists of tensors at the sizes where a block's share changes: a list that the GPU
holds at once in blocks of 256 elements and one element more, and sums of squares
over more than 152 x 32 blocks of 2048; the loss of rounding is that of
test_gpu_lists.py.
"""

import pytest

import test_gpu_lists
from sunlightlb_gb300.warmstart import Kernels

pytestmark = pytest.mark.gpu

FITS = 152 * 8 * 256


@pytest.mark.parametrize("sizes", [[1], [FITS], [FITS + 1], [300, FITS - 600, 257], [FITS, 1, 255, 256, 257], [27648], [500_000] * 7])
def test_adam_squares_and_scale(gpu, monkeypatch, sizes):
    monkeypatch.setattr(test_gpu_lists, "SIZES", sizes)
    test_gpu_lists.test_adam_squares_and_scale(gpu)


@pytest.mark.parametrize("n", [152 * 32 * 2048, 152 * 32 * 2048 + 1, 25_000_003, 70_000_001])
def test_squares_of_large_tensors(gpu, n):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    g = torch.randint(-3, 4, (n,), device="cuda", dtype=torch.int8).float()  # sums are exact
    state = torch.tensor([0.5, 2.0, 0.0], device="cuda", dtype=torch.float64)
    k.nn_sqsum(g.data_ptr(), n, state.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert float(state[0]) == 0.5 + float((g.double() ** 2).sum())
