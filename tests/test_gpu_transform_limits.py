"""The Legendre sums of the transform API at the ends of their launch shapes."""

import pytest

from test_gpu_step_kernels import test_legendre_api_against_fp64_sums as _sums

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("B,J,N,C", [(80, 436, 15, 1), (80, 440, 15, 1), (80, 700, 15, 1),
                                     (40, 1100, 15, 2)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_few_columns_of_many_latitudes(torch, B, J, N, C, dtype):
    """Large batches of one or two columns on more latitudes than a block's
    shared memory holds as table rows: the bounds of the smaller shapes."""
    _sums(torch, B, J, N, C, True, dtype)
