"""The fused step where its plans and buffers meet a limit: grids that fill a
block's shared memory."""

import ctypes as C

import pytest

from test_gpu_step_kernels import (_grid_stepper,
                                   test_legendre_kernels_against_fp64_sums as _legendre_sums)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("I,J,N,K,nmem", [
    (256, 128, 112, 4, 43), (256, 128, 127, 20, 1), (256, 128, 127, 20, 8),   # one state buffer
    (128, 370, 54, 5, 1), (256, 252, 69, 9, 3), (256, 252, 69, 2, 96)])       # two tables
def test_fp64_legendre_on_grids_that_fill_shared_memory(torch, I, J, N, K, nmem):
    """k_anal and k_synth in FP64 where the synthesis has room for one state
    buffer of several members, or for two of its three tables: the bounds of the
    smaller grids."""
    _legendre_sums(torch, I, J, N, K, nmem, "fp64")


@pytest.mark.parametrize("precision,nlat", [("fp64", 1000), ("fp32", 2000)])
def test_a_grid_beyond_shared_memory_is_refused(torch, precision, nlat):
    """Tables over 227 KB: LBM_ERR_ARG before any launch."""
    from lbm_isca_gb300._lib import LBM_ERR_ARG, StepperDesc, lib
    stp = _grid_stepper(torch, 64, 32, 30, 2, 1, precision)
    d = StepperDesc.from_buffer_copy(stp.desc())
    d.nlat = nlat
    s = C.c_void_p(stp.stream.cuda_stream)
    ctl = stp._ctl([(stp._dts[0], False, 0)])
    assert lib().lbm_stepper_prime(C.byref(d), s) == LBM_ERR_ARG
    assert lib().lbm_stepper_run(C.byref(d), ctl, 1, s) == LBM_ERR_ARG
