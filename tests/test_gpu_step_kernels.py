"""Kernels of the fused step at the edges of their tiles and dispatch rules,
each against another route to the same numbers."""

import ctypes as C

import numpy as np
import pytest

from lbm_isca_gb300 import configs

pytestmark = pytest.mark.gpu

GRIDS = {"T21": (64, 32, 21), "T42": (128, 64, 42), "T85": (256, 128, 85)}


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _stepper(torch, grid, K, nmem, precision, **kw):
    """Stepper on a humid solid-body state with a random spectral state."""
    from lbm_isca_gb300 import Config
    from lbm_isca_gb300.ensemble import make_ensemble_model
    I, J, N = GRIDS[grid]
    sigm = configs.equal_sigma_half_levels(K)
    bs = configs.solid_body_basic_state(I, J, sigm)
    mu, _ = configs.gaussian_latitudes(J)
    bs.q = np.broadcast_to(0.01 * (1.0 - mu * mu)[:, None, None], bs.t.shape).copy()
    cfg = dict(configs.plain_damping(K), **kw)
    m, _, _ = make_ensemble_model(bs, nmem, Config(precision=precision, **cfg), device="gb300",
                                  nlon=I, nlat=J, nmax=N, sigm=sigm)
    stp = m.stepper()
    stp.set_timesteps([600.0])
    g = torch.Generator().manual_seed(11)
    M = N + 1

    def spec(scale, k=True):
        z = torch.randn((nmem, M, M) + ((K,) if k else ()) + (2,), generator=g,
                        dtype=torch.float64) * scale
        z[:, 0, ..., 1] = 0.0
        return torch.view_as_complex(z).cuda()

    scales = {"vor": 1e-6, "div": 1e-7, "t": 0.1, "q": 1e-5}
    a = {k: spec(s) for k, s in scales.items()}
    b = {k: spec(s) for k, s in scales.items()}
    a["pi"] = spec(1e-4, k=False)
    ps = lambda: torch.randn((nmem, J, I), generator=g, dtype=torch.float64).cuda()  # noqa: E731
    stp.load(a, b, ps(), ps())
    torch.cuda.synchronize()
    return stp


def _launch(torch, stp, kernel, desc=None, ps_mode=0):
    from lbm_isca_gb300._lib import check, lib
    ctl = stp._ctl([(stp._dts[0], False, ps_mode)])
    check(lib().lbm_stepper_launch(C.byref(stp.desc() if desc is None else desc), ctl, kernel,
                                   C.c_void_p(stp.stream.cuda_stream)), "launch")
    torch.cuda.synchronize()


def _rel(x, y):
    return float((x - y).abs().max() / y.abs().max())


@pytest.mark.parametrize("grid,K,nmem", [("T21", 4, 1), ("T21", 9, 3), ("T42", 2, 2),
                                         ("T42", 17, 1), ("T85", 5, 1)])
@pytest.mark.parametrize("ps_mode", [0, 1, 2])
def test_fp64_split_grid_part_equals_the_one_kernel_form(torch, grid, K, nmem, ps_mode):
    """k_ifft, k_alg, k_ffft against k_grid (no grid-row buffers): the same
    algebra in another order.  Per output field, double rounding (1.1e-16)
    times the two FFTs' log2(I) stages and the temperature equation's
    cancellation (250 K against 0.1 K) stays below 1e-11 of the largest value."""
    from lbm_isca_gb300._lib import StepperDesc
    stp = _stepper(torch, grid, K, nmem, "fp64")
    assert stp.grid6 is not None and stp.launches_per_step() == 6
    ps0 = stp.psa.clone(), stp.psb.clone()
    _launch(torch, stp, 0, ps_mode=ps_mode)
    got = [x.clone() for x in (stp.af, stp.afs, stp.psa, stp.psb)]
    for x, y in zip((stp.psa, stp.psb), ps0):
        x.copy_(y)
    stp.af.zero_()
    stp.afs.zero_()
    d = StepperDesc.from_buffer_copy(stp.desc())
    d.grid6 = d.grid9 = None
    _launch(torch, stp, 0, desc=d, ps_mode=ps_mode)
    for f in range(7):
        assert _rel(got[0][..., f], stp.af[..., f]) < 1e-11
    for f in range(2):
        assert _rel(got[1][..., f], stp.afs[..., f]) < 1e-11
    assert _rel(got[2], stp.psa) < 1e-12 and _rel(got[3], stp.psb) < 1e-12
