"""The fused step where its plans and buffers meet a limit: grids that fill a
block's shared memory, steppers of different sizes side by side, arrays off their
elements' alignment, FP64 without grid rows."""

import ctypes as C
import threading

import pytest

from lbm_isca_gb300 import configs
from test_gpu_step_kernels import (_grid_stepper, _launch, _noise, _rel, _stepper,
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


SIDE_BY_SIDE = [  # grid, levels, members of two groups; each kernel's launches need the
                  # more shared memory in the first group of one of them
    [("T42", 20, 128), ("T42", 20, 8)], [("T42", 20, 32), ("T42", 20, 1)],
    [("T42", 20, 1), ("T42", 20, 32)], [("T42", 20, 32), ("T21", 20, 48)],
    [("T42", 20, 128), ("T85", 40, 1)]]
GRIDS = {"T21": (64, 32, 21), "T42": (128, 64, 42), "T85": (256, 128, 85)}


@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16split"])
@pytest.mark.parametrize("sizes", SIDE_BY_SIDE)
def test_groups_of_any_order_and_size(torch, sizes, precision):
    """One graph records the steps of all groups: no group's launches depend on
    the plans of the others.  Each group equals itself alone."""
    from lbm_isca_gb300.grouped import GroupedEnsemble
    groups = []
    for name, K, E in sizes:
        I, J, N = GRIDS[name]
        sigm = configs.equal_sigma_half_levels(K)
        heats, _ = configs.ensemble_heating(I, J, sigm, E, seed=5)
        groups.append(dict(nlon=I, nlat=J, nmax=N, sigm=sigm, heats=heats,
                           basic_state=configs.solid_body_basic_state(I, J, sigm),
                           config=configs.plain_damping(K)))
    together = GroupedEnsemble(groups, precision=precision, tune=False).run(4)
    assert together.check_finite()
    for g, state in zip(groups, together.spectral_states()):
        alone = GroupedEnsemble([g], precision=precision, tune=False).run(4)
        assert float(state["t"].abs().max()) > 0
        for k, x in alone.spectral_states()[0].items():
            assert torch.equal(x, state[k]), k


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_steppers_on_two_threads(torch, precision):
    """Two host threads step ensembles of different sizes, launch by launch:
    the same state as one after the other."""
    steps = [(600.0, False)] * 150
    pair = [_grid_stepper(torch, 128, 64, 42, 20, E, precision) for E in (32, 1)]
    g = torch.Generator().manual_seed(4)
    heat = torch.zeros((43, 43, 20), dtype=torch.complex128)
    heat[:6, 5:9] = torch.view_as_complex(
        torch.randn((6, 4, 20, 2), generator=g, dtype=torch.float64)) * 1e-6
    heat[0] = heat[0].real.clone()
    for s in pair:
        s.set_forcing(frc_t=heat.cuda())

    def start():
        for s in pair:
            s.load_zero()
        torch.cuda.synchronize()

    def state():
        torch.cuda.synchronize()
        return [s.sa3.clone() for s in pair]

    start()
    for s in pair:
        s.run(steps, use_graph=False)
    want = state()
    for x in want:
        assert bool(torch.isfinite(torch.view_as_real(x)).all()) and float(x.abs().max()) > 0
    start()
    errors = []

    def work(s):
        try:
            s.run(steps, use_graph=False)
        except Exception as exc:
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(s,)) for s in pair]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, b in zip(state(), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("I,J,N,K,nmem", [(64, 32, 21, 7, 1), (128, 64, 42, 20, 9),
                                          (128, 50, 31, 2, 3)])
@pytest.mark.parametrize("precision", ["fp64", "bf16x3"])
def test_surface_rows_off_their_alignment(torch, I, J, N, K, nmem, precision):
    """afs on the alignment of its real type only: k_anal reads the same values."""
    from lbm_isca_gb300._lib import StepperDesc
    if precision == "bf16x3" and (K % 2 or J % 16):
        pytest.skip("no tensor-core form")
    stp = _grid_stepper(torch, I, J, N, K, nmem, precision)
    _noise(torch, stp.af, 1)
    _noise(torch, stp.afs, 2)
    _launch(torch, stp, 1)
    want = stp.tend.clone(), stp.tends.clone()
    assert float(want[1].abs().max()) > 0
    r = torch.view_as_real(stp.afs).reshape(-1)
    buf = torch.empty(r.numel() + 1, device="cuda", dtype=r.dtype)
    buf[1:] = r
    stp.tend.zero_()
    stp.tends.zero_()
    d = StepperDesc.from_buffer_copy(stp.desc())
    d.afs = buf[1:].data_ptr()
    _launch(torch, stp, 1, desc=d)
    assert torch.equal(stp.tend, want[0]) and torch.equal(stp.tends, want[1])


@pytest.mark.parametrize("precision,tc_off,name,bytes_off", [
    ("fp64", 0, "sf", 8), ("fp64", 0, "af", 8), ("fp32", 0, "grid9", 8), ("fp32", 0, "sfs", 4),
    ("fp32", 0, "dft", 4), ("fp32", 0, "afs", 4), ("bf16x3", 7, "afs", 4),
    ("bf16split", 0, "sa3", 8)])
def test_alignment_that_kernels_need_is_checked(torch, precision, tc_off, name, bytes_off):
    """LBM_ERR_ARG before any launch."""
    from lbm_isca_gb300._lib import LBM_ERR_ARG, StepperDesc, lib
    stp = _grid_stepper(torch, 64, 32, 21, 4, 1, precision)
    d = StepperDesc.from_buffer_copy(stp.desc())
    if stp.legendre:
        d.tc_off = tc_off
    setattr(d, name, getattr(d, name) + bytes_off)
    s = C.c_void_p(stp.stream.cuda_stream)
    ctl = stp._ctl([(stp._dts[0], False, 0)])
    assert lib().lbm_stepper_prime(C.byref(d), s) == LBM_ERR_ARG
    assert lib().lbm_stepper_run(C.byref(d), ctl, 1, s) == LBM_ERR_ARG


def test_fp64_run_without_grid_rows(torch, monkeypatch):
    """EnsembleStepper past the limit of its grid rows: the one-kernel grid part
    over 20 steps equals the split one to the round-off that the steps carry
    along (1e-10 of a field's largest value)."""
    from lbm_isca_gb300.stepper import EnsembleStepper
    split = _stepper(torch, "T42", 20, 2, "fp64")
    monkeypatch.setattr(EnsembleStepper, "GRID_ROWS_BYTES", 0)
    whole = _stepper(torch, "T42", 20, 2, "fp64")
    assert split.launches_per_step() == 6 and whole.launches_per_step() == 4
    for s in (split, whole):
        s.run([(600.0, True)] + [(600.0, False)] * 20)
        torch.cuda.synchronize()
        assert s.check_finite()
    for f in range(4):
        assert _rel(whole.sa3[:, f], split.sa3[:, f]) < 1e-10
