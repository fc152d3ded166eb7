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
    torch.cuda.synchronize()          # the test writes its inputs on another stream
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


def _grid_stepper(torch, I, J, N, K, nmem, precision):
    """Stepper on any grid (its arrays only: the state is set by the test)."""
    from lbm_isca_gb300 import Config
    from lbm_isca_gb300.ensemble import make_ensemble_model
    sigm = configs.equal_sigma_half_levels(K)
    cfg = dict(configs.plain_damping(max(K, 2)), ddragv=None, ddragd=None, ddragt=None)
    m, _, _ = make_ensemble_model(configs.solid_body_basic_state(I, J, sigm), nmem,
                                  Config(precision=precision, **cfg),
                                  device="gb300", nlon=I, nlat=J, nmax=N, sigm=sigm)
    stp = m.stepper()
    stp.set_timesteps([600.0])
    stp.load_zero()
    torch.cuda.synchronize()
    return stp


def _full_tables(torch, stp):
    """P, H [m][n][j] in FP64 from the stepper's northern, working-precision rows."""
    M, JH = stp.M, stp.J // 2
    sign = torch.where((stp.pn - stp.pm) % 2 == 0, 1.0, -1.0).double()[:, None]
    out = []
    for t, s in ((stp.symp.double(), sign), (stp.symh.double(), -sign)):
        T = torch.zeros((M, M, stp.J), device=t.device, dtype=torch.float64)
        T[stp.pm, stp.pn, :JH] = t
        T[stp.pm, stp.pn, JH:] = (s * t).flip(1)
        out.append(T)
    return out


def _noise(torch, like, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(tuple(like.shape) + (2,), generator=g, device="cuda", dtype=torch.float64)
    like.copy_(torch.view_as_complex(x).to(like.dtype))


SHAPES = [  # I, J, N, K, members: odd level counts, one level, J/2 odd, N odd and even,
            # level chunks with remainders, one and many members, units beyond the SMs
    (64, 32, 21, 1, 1), (64, 32, 21, 20, 1), (64, 30, 19, 5, 3), (64, 32, 21, 40, 9),
    (128, 64, 42, 17, 2), (128, 64, 42, 20, 13), (128, 50, 31, 2, 1), (256, 128, 85, 9, 2),
    (256, 128, 85, 40, 1), (64, 6, 3, 7, 40)]


@pytest.mark.parametrize("I,J,N,K,nmem", SHAPES)
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_legendre_kernels_against_fp64_sums(torch, I, J, N, K, nmem, precision):
    """k_anal and k_synth against plain FP64 contractions of the same working-
    precision tables and rows.  Bound per value: the rounding of a sum of n <= 2 J
    products (and the three or four operations around it), (n + 8) u times the
    sum of the products' magnitudes, u the unit roundoff, plus gradual underflow:
    half the least subnormal per operation, times m (near the poles P and H of
    large m fall below the least normal number)."""
    stp = _grid_stepper(torch, I, J, N, K, nmem, precision)
    u, tiny = (2.0 ** -24, 2.0 ** -150) if precision == "fp32" else (2.0 ** -53, 1e-300)
    P, H = _full_tables(torch, stp)
    m = torch.arange(stp.M, device="cuda", dtype=torch.float64)
    im = (1j * m)[None, :, None, None]
    pm, pn = stp.pm, stp.pn

    def mul(eq, T, X):
        return torch.complex(torch.einsum(eq, T, X.real.contiguous()),
                             torch.einsum(eq, T, X.imag.contiguous()))

    def check(got, want, size, terms):
        # size: sum of magnitudes, the largest of its (Re, Im) parts
        err = torch.view_as_real(got.to(torch.complex128) - want).abs().amax(-1)
        lim = (terms + 8) * (u * size + (1.0 + N) * tiny)
        assert bool((err <= lim).all()), float((err / lim).max())

    # ---- analysis
    _noise(torch, stp.af, 1)
    _noise(torch, stp.afs, 2)
    for t in (stp.tend, stp.tends):
        t.zero_()
    _launch(torch, stp, 1)
    af = stp.af.to(torch.complex128)                    # [E][M][J][K][7]
    ab = af.abs()
    fu, fv, ke, t, xv, q, yv = af.unbind(-1)
    afu, afv, ake, at, axv, aq, ayv = ab.unbind(-1)
    A = lambda T, X: mul("mnj,emjk->emnk", T, X)         # noqa: E731
    B = lambda T, X: torch.einsum("mnj,emjk->emnk", T.abs(), X)     # noqa: E731
    nn = stp.nn1a.double()[None, None, :, None]
    mm = m[None, :, None, None]
    want = [im * A(P, fv) + A(H, fu), im * A(P, fu) - A(H, fv) + nn * A(P, ke),
            A(P, t) + A(H, xv), A(P, q) + A(H, yv)]
    size = [mm * B(P, afv) + B(H, afu), mm * B(P, afu) + B(H, afv) + nn * B(P, ake),
            B(P, at) + B(H, axv), B(P, aq) + B(H, ayv)]
    for f in range(4):
        check(stp.tend[:, f], want[f][:, pm, pn], size[f][:, pm, pn], J)
    for f in range(2):
        X = stp.afs.to(torch.complex128)[..., f]
        check(stp.tends[:, f], mul("mnj,emj->emn", P, X)[:, pm, pn],
              torch.einsum("mnj,emj->emn", P.abs(), X.abs())[:, pm, pn], J)

    # ---- synthesis
    _noise(torch, stp.sa3, 3)
    _noise(torch, stp.sas, 4)
    for t in (stp.sf, stp.sfs):
        t.zero_()
    _launch(torch, stp, 3)

    def rect(x):                                         # [E][NS] + tail -> [E][M][M] + tail
        r = torch.zeros((nmem, stp.M, stp.M) + tuple(x.shape[2:]), device="cuda",
                        dtype=torch.complex128)
        r[:, pm, pn] = x.to(torch.complex128)
        return r

    S = lambda T, X: mul("mnj,emnk->emjk", T, X)         # noqa: E731
    Q = lambda T, X: torch.einsum("mnj,emnk->emjk", T.abs(), X.abs())   # noqa: E731
    il = stp.invlap.double()[None, None, :, None]

    def winds(psi, chi):
        return ([im * S(P, chi) - S(H, psi), im * S(P, psi) + S(H, chi)],
                [mm * Q(P, chi) + Q(H, psi), mm * Q(P, psi) + Q(H, chi)])

    vo, dv, tt, qq = (rect(stp.sa3[:, f]) for f in range(4))
    w, wz = winds(vo * il, dv * il)
    want = w + [S(P, x) for x in (vo, dv, tt, qq)]
    size = wz + [Q(P, x) for x in (vo, dv, tt, qq)]
    for f in range(6):
        check(stp.sf[..., f], want[f], size[f], N + 1)
    pi, psi, chi, ds = (rect(stp.sas[:, f])[..., None] for f in range(4))
    w, wz = winds(psi, chi)
    want = [S(P, pi), S(H, pi)] + w + [S(P, ds)]
    size = [Q(P, pi), Q(H, pi)] + wz + [Q(P, ds)]
    for f in range(5):
        check(stp.sfs[..., f], want[f][..., 0], size[f][..., 0], N + 1)
    assert int(stp.err.item()) == 0


IMPL_SHAPES = [  # I, J, N, K, members: one coefficient per share and many, one level, the
                 # most levels, shares that cross from one n of a pair to the other, N odd and even
    (64, 32, 21, 1, 1), (64, 32, 21, 64, 1), (64, 6, 3, 7, 40), (128, 50, 31, 2, 3),
    (128, 64, 42, 20, 1), (128, 64, 42, 17, 30), (256, 128, 85, 9, 2)]


@pytest.mark.parametrize("I,J,N,K,nmem", IMPL_SHAPES)
@pytest.mark.parametrize("vdiff", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_implicit_kernel_against_fp64_formula(torch, I, J, N, K, nmem, vdiff, precision):
    """k_implicit against the update written out in FP64 on the same operators.
    Each result is a sum of products along a path of at most 4 K + 40 rounded
    operations: that many u times the same formula on magnitudes.  Arrays moved
    off their element alignment take the narrow accesses: the same bits."""
    from lbm_isca_gb300._lib import StepperDesc
    stp = _grid_stepper(torch, I, J, N, K, nmem, precision)
    u = 2.0 ** -24 if precision == "fp32" else 2.0 ** -53
    for x, seed, scale in ((stp.sa3, 1, 1.0), (stp.sb3, 2, 1.0), (stp.tend, 3, 1e-3),
                           (stp.tends, 4, 1e-3)):
        _noise(torch, x, seed)
        x.mul_(scale)
    stp.vd_on = [int(vdiff)] * 4
    g = torch.Generator(device="cuda").manual_seed(5)
    stp.vdm = torch.randn((1, 4, K, K), generator=g, device="cuda",
                          dtype=torch.float64).mul(0.1).to(stp.minv.dtype)
    stp._desc = None
    dt, K1 = 600.0, K + 1
    vert = stp.vert.double().reshape(-1, K1)[:, :K]
    dsig, alpha, w3 = vert[0], vert[2], vert[3]
    rdlog3, ralpha, ktref, gg = vert[6], vert[7], vert[9], vert[11]
    pm, pn = stp.pm, stp.pn
    cplx = lambda x: x.to(torch.complex128)                       # noqa: E731
    prev = [cplx(stp.sa3[:, f]) for f in range(4)]
    b = [cplx(stp.sb3[:, f]) for f in range(4)]
    w = [cplx(stp.tend[:, f]) for f in range(4)]
    wpi, pi = (cplx(stp.tends[:, f]) for f in range(2))
    tab = lambda x: x.double().reshape(stp.M, K)[pn]              # noqa: E731
    ktt, kd, kv, kq = tab(stp.ktt), tab(stp.kd), tab(stp.kv), tab(stp.kq)
    lap, il = stp.lap.double()[pn][:, None], stp.invlap.double()[pn][:, None]
    minv = stp.minv[0].double()[pn]
    vdm, gam = stp.vdm[0].double(), float(torch.tensor(stp.robert, dtype=stp.minv.dtype))

    def update(prev, b, w, wpi, pi, lap, il, minv, vdm, s):
        """s = -1: the update; s = +1 with magnitudes: its bound."""
        wdx = b[2] + dt * (b[2] * ktt + w[2])
        run = torch.cumsum(wdx * rdlog3, -1) - wdx * rdlog3 if s < 0 else \
            torch.cumsum(wdx * rdlog3, -1)
        bt = 2 * dt * ktt
        phi = ralpha * wdx + run + (1 + bt) * gg * (pi + dt * wpi)[..., None]
        ad = dt * kd
        rhs = b[1] + b[1] * (ad + bt + ad * bt) + dt * ((1 + bt) * w[1] + s * lap * phi)
        dbar = torch.einsum("slk,esl->esk", minv.to(rhs.dtype), rhs)
        x = dsig * dbar
        after = x.flip(-1).cumsum(-1).flip(-1) + (s * x if s < 0 else 0)
        damp = lambda y, c: y + s * y * (c / (1 + c))             # noqa: E731
        t = damp(b[2] + 2 * dt * (w[2] + s * ktref * (alpha * dbar + w3 * after)), bt)
        npi = pi + 2 * dt * (wpi + s * x.sum(-1))
        new = [damp(b[0] + 2 * dt * w[0], 2 * dt * kv), 2 * dbar + s * b[1], t,
               damp(b[3] + 2 * dt * w[3], 2 * dt * kq)]
        if vdiff:
            for f in range(4):
                on = ((pn >= 2) | torch.tensor(f >= 2, device="cuda"))[:, None]
                new[f] = new[f] + on * torch.einsum("lk,esl->esk", vdm[f].to(rhs.dtype), new[f])
        old = [a + gam * (b_ + s * 2 * a + n) for a, b_, n in zip(prev, b, new)]
        sv, sd = (new[0] * dsig).sum(-1), (new[1] * dsig).sum(-1)
        il0 = il[:, 0]
        return new, old, [npi, sv * il0, sd * il0, sd]

    a = lambda xs: [x.abs() for x in xs]                          # noqa: E731
    want = update(prev, b, w, wpi, pi, lap, il, minv, vdm, -1)
    size = update(a(prev), a(b), a(w), wpi.abs(), pi.abs(), lap.abs(), il.abs(), minv.abs(),
                  vdm.abs(), 1)
    state = [x.clone() for x in (stp.sa3, stp.sb3)]
    _launch(torch, stp, 2)
    got = stp.sa3, stp.sb3, stp.sas
    for gx, wx, sx in zip(got, want, size):
        for f in range(4):
            err = (cplx(gx[:, f]) - wx[f]).abs()
            lim = (4 * K + 40) * u * sx[f] + 1e-300
            assert bool((err <= lim).all()), (f, float((err / lim).max()))
    assert int(stp.err.item()) == 0

    first = [x.clone() for x in got]
    moved, views = [], []
    for x in (state[0], state[1], stp.tend):
        r = torch.view_as_real(x).reshape(-1)
        buf = torch.empty(r.numel() + 1, device="cuda", dtype=r.dtype)
        buf[1:] = r
        moved.append(buf)
        views.append(buf[1:])
    d = StepperDesc.from_buffer_copy(stp.desc())
    d.sa3, d.sb3, d.tend = (v.data_ptr() for v in views)
    stp.sas.zero_()
    _launch(torch, stp, 2, desc=d)
    for v, f in zip(views[:2], first):
        assert torch.equal(v, torch.view_as_real(f).reshape(-1))
    assert torch.equal(stp.sas, first[2])


@pytest.mark.parametrize("B,J,N,C", [(1, 64, 42, 20), (1, 6, 3, 1), (2, 50, 31, 17), (1, 64, 42, 35),
                                     (3, 34, 21, 40), (1, 128, 85, 65), (1, 64, 42, 1),
                                     (40, 64, 42, 21), (1, 64, 42, 1000)])
@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_legendre_api_against_fp64_sums(torch, B, J, N, C, two, dtype):
    """The Legendre sums of the transform API over column chunks with
    remainders, one column, row tiles that end early and both block sizes, on
    tables without symmetry.  Bound per value: (terms + 8) u times the sum of
    the products' magnitudes."""
    import lbm_isca_gb300.ops      # noqa: F401  (registers the operators)
    rt = getattr(torch, dtype)
    ct = torch.complex64 if dtype == "float32" else torch.complex128
    u, M = torch.finfo(rt).eps / 2, N + 1
    g = torch.Generator(device="cuda").manual_seed(B + J + C)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)   # noqa: E731
    ta, tb = rnd(M, M, J).to(rt), rnd(M, M, J).to(rt)
    fac = [rnd(M).to(rt) for _ in range(3)]
    field = lambda *s: torch.view_as_complex(rnd(*s, 2)).to(ct)     # noqa: E731
    m = torch.arange(M, device="cuda", dtype=torch.float64)[None, :, None, None]
    tri = (torch.arange(M, device="cuda")[None, :] >= torch.arange(M, device="cuda")[:, None])
    D = lambda x: x.to(torch.complex128 if x.is_complex() else torch.float64)   # noqa: E731

    def mul(eq, T, X):
        return torch.complex(torch.einsum(eq, D(T), D(X).real.contiguous()),
                             torch.einsum(eq, D(T), D(X).imag.contiguous()))

    def check(got, want, size, terms):
        err = torch.view_as_real(D(got) - want).abs().amax(-1)
        assert bool((err <= (terms + 8) * u * size + 1e-300).all())

    fa, fb = field(B, M, J, C), field(B, M, J, C)
    got = torch.ops.lbm_gb300.legendre_analysis(fa, ta, 1, fb if two else None,
                                                tb if two else None, 0, -1.5, fac[0])
    A = lambda T, X: mul("mnj,bmjc->bmnc", T, X)         # noqa: E731
    Z = lambda T, X: torch.einsum("mnj,bmjc->bmnc", D(T).abs(), D(X).abs())   # noqa: E731
    want, size = 1j * m * A(ta, fa), m * Z(ta, fa)
    if two:
        want, size = want - 1.5 * A(tb, fb), size + 1.5 * Z(tb, fb)
    nf = D(fac[0])[None, None, :, None] * tri[None, :, :, None]
    check(got, want * nf, size * nf.abs(), 2 * J)

    sa, sb = field(B, M, M, C), field(B, M, M, C)
    got = torch.ops.lbm_gb300.legendre_synthesis(sa, ta, 0, fac[1], sb if two else None,
                                                 tb if two else None, 1, fac[2], 0.5)
    tr = tri[None, :, :, None]
    S = lambda T, X: mul("mnj,bmnc->bmjc", T, X)         # noqa: E731
    Q = lambda T, X: torch.einsum("mnj,bmnc->bmjc", D(T).abs(), D(X).abs())   # noqa: E731
    x = D(sa) * D(fac[1])[None, None, :, None] * tr
    want, size = S(ta, x), Q(ta, x)
    if two:
        x = 0.5j * m * D(sb) * D(fac[2])[None, None, :, None] * tr
        want, size = want + S(tb, x), size + Q(tb, x)
    check(got, want, size, 2 * M)


@pytest.mark.parametrize("K", [2, 7, 20, 64])
@pytest.mark.parametrize("linear", [False, True])
def test_tendency_kernel_against_oracle(torch, K, linear):
    """Grid tendencies at level counts that divide a block's threads and that
    do not, against the oracle (as at 20 levels: 1e-10 of the largest value)."""
    import types
    from lbm_isca_gb300 import LBM, Config, Spectral, VerticalGrid
    from oracle import lbm_oracle as orc
    from lbm_isca_gb300.state import State
    I, J, N = 64, 32, 21
    sigm = configs.equal_sigma_half_levels(K)
    bs = configs.solid_body_basic_state(I, J, sigm)
    mu, _ = configs.gaussian_latitudes(J)
    bs.q = np.broadcast_to(0.01 * (1.0 - mu * mu)[:, None, None], bs.t.shape).copy()
    cfg = dict(configs.plain_damping(K), strictly_linear=linear)
    m = LBM(bs, Spectral(nlon=I, nlat=J, nmax=N, device="gb300"),
            VerticalGrid(sigm=sigm, device="gb300"), Config(**cfg))
    tr, lv = orc.SphericalTransform(I, J, N), orc.SigmaLevels(sigm)
    om = orc.OracleModel(tr, lv, bs, orc.RunConfig(**cfg))
    rng = np.random.default_rng(K)
    u, v = tr.vordiv_to_uv(*tr.uv_to_vordiv(*rng.normal(size=(2, J, I, K))))
    wave = lambda x: tr.wave_to_grid(tr.grid_to_wave(x))          # noqa: E731
    f = types.SimpleNamespace(u=u, v=v, t=wave(rng.normal(size=(J, I, K))),
                              q=wave(1e-3 * rng.normal(size=(J, I, K))),
                              ps=0.5 * wave(rng.normal(size=(J, I))))
    heat = configs.elliptic_heating(I, J, sigm)
    got = m.dyn.tendencies(State(bs.ps, u=f.u, v=f.v, t=f.t, q=f.q, ps=f.ps, device="gb300"),
                           frc_t=heat)
    ref = orc.tendencies(tr, lv, om.bt, orc.GridState(np.asarray(bs.ps), f.u, f.v, f.t, f.q, f.ps),
                         frc_t=heat, strictly_linear=linear)
    for a, b in zip(got, ref):
        a = a.detach().cpu().numpy()
        assert np.abs(a - b).max() < 1e-10 * np.abs(b).max()


@pytest.mark.parametrize("K", [2, 7, 33, 64])
def test_adjoint_kernels_are_the_transposes(torch, K):
    """<A x, y> = <x, A^T y> for the grid tendencies (linearised) and the
    implicit update with vertical diffusion, at level counts that divide a
    block's threads and that do not.  Both sides are sums of products rounded a
    few hundred times: 1e-13 of |A x| |y|."""
    from lbm_isca_gb300.adjoint import TimeStep, spec_dot, state_dot
    from test_adjoint import _Rand, _model
    m, _ = _model(K, vdifv=1.0e3, vdifd=1.0e3, vdift=1.0e3, vdifq=2.0e3)
    st, r = TimeStep(m), _Rand(torch, K, K=K)
    norm = lambda xs: float(sum(spec_dot(x, x) for x in xs)) ** 0.5      # noqa: E731

    def check(ax, y, rhs):
        lhs = float(sum(spec_dot(a, b) for a, b in zip(ax, y)))
        assert abs(lhs - float(rhs)) < 1e-13 * norm(ax) * norm(y)

    ga, dx = r.state(st), r.state(st)
    aw = [r.spec(), r.spec(), r.spec(), r.spec(False), r.spec()]
    check(st.tangent_tendencies(ga, dx), aw, state_dot(dx, st.adjoint_tendencies(ga, aw)))
    keys = ("vor", "div", "t", "pi", "q")
    p, y = ({k: r.spec(k != "pi") for k in keys} for _ in range(2))
    w = [r.spec(k != "pi") for k in keys]
    new = m.integ.step(1200.0, p, w)
    ap, aw2 = st._implicit_adjoint(1200.0, y)
    check([new[k] for k in keys], [y[k] for k in keys],
          sum(spec_dot(p[k], ap[k]) for k in keys)
          + sum(spec_dot(wi, aw2[k]) for wi, k in zip(w, keys)))


@pytest.mark.parametrize("grid,K", [("T21", 2), ("T21", 21), ("T21", 64), ("T42", 20),
                                    ("T42", 7)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ps_mode", [0, 2])
def test_column_segments_equal_whole_columns(torch, grid, K, precision, ps_mode):
    """k_alg of one member (columns cut into level segments) against the same
    member in an ensemble large enough for whole columns: the same bits in FP32,
    rounding of the column sums (1e-13 of the largest value) in FP64."""
    one = _stepper(torch, grid, K, 1, precision)
    many = _stepper(torch, grid, K, 20, precision)
    for name in ("sf", "sfs", "psa", "psb"):
        getattr(many, name).copy_(getattr(one, name).expand_as(getattr(many, name)))
    for s in (one, many):
        s.grid9.zero_()
        _launch(torch, s, 0, ps_mode=ps_mode)
    for name in ("grid9", "psa", "psb"):
        a = getattr(one, name)[0]
        b = getattr(many, name).reshape(20, *a.shape)[19]
        assert float(a.abs().max()) > 0
        if precision == "fp32":
            assert torch.equal(a, b)
        else:
            assert _rel(a, b) < 1e-13


@pytest.mark.parametrize("I,J,N,K,nmem", [(64, 32, 21, 1, 1), (64, 32, 21, 20, 2), (64, 6, 3, 7, 9),
                                          (128, 64, 42, 17, 3), (128, 64, 63, 3, 1),
                                          (128, 64, 42, 64, 1), (256, 128, 85, 9, 2),
                                          (256, 128, 127, 5, 1)])
def test_longitude_analysis_against_fp64_sums(torch, I, J, N, K, nmem):
    """k_fdft against FP64 transforms of the same rows: level chunks with
    remainders, one level, the most wavenumbers.  Bound per value: I + 16
    operations on terms that sum to the row's magnitudes (times m for the
    rows combined with a derivative)."""
    stp = _grid_stepper(torch, I, J, N, K, nmem, "fp32")
    u = 2.0 ** -24
    g = torch.Generator(device="cuda").manual_seed(I + K)
    stp.grid9.copy_(torch.randn(stp.grid9.shape, generator=g, device="cuda", dtype=torch.float64))
    stp.af.zero_()
    stp.afs.zero_()
    _launch(torch, stp, 6)
    x = stp.grid9.double()                               # [E][J][2 + 9K][I]
    X = torch.fft.rfft(x, dim=-1)[..., :stp.M]
    A = x.abs().sum(-1, keepdim=True).expand_as(X)
    jf = stp.jfac.double().reshape(4, J)
    wg, wd = (jf[k][None, :, None, None] / I for k in (0, 1))    # gw, gw del cos
    m = torch.arange(stp.M, device="cuda", dtype=torch.float64)
    rows = [X[:, :, 2 + f::9] for f in range(9)]         # gt xu g yu fu fv ke xv yv
    mag = [A[:, :, 2 + f::9] for f in range(9)]
    want = [wd * rows[4], wd * rows[5], wg * rows[6], wg * rows[0] - wd * 1j * m * rows[1],
            wd * rows[7], wg * rows[2] - wd * 1j * m * rows[3], wd * rows[8]]
    size = [wd * mag[4], wd * mag[5], wg * mag[6], wg * mag[0] + wd * m * mag[1],
            wd * mag[7], wg * mag[2] + wd * m * mag[3], wd * mag[8]]
    for f in range(7):
        got = stp.af[..., f].to(torch.complex128).permute(0, 2, 3, 1)      # [E][J][K][M]
        assert bool(((got - want[f]).abs() <= (I + 16) * u * size[f]).all()), f
    for f in range(2):
        got = stp.afs[..., f].to(torch.complex128).permute(0, 2, 1)
        assert bool(((got - (wg * X)[:, :, f]).abs() <= (I + 16) * u * (wg * A)[:, :, f]).all())


@pytest.mark.parametrize("I,J,N,K,nmem", [(64, 32, 21, 1, 1), (64, 32, 21, 20, 12), (64, 6, 31, 7, 1),
                                          (128, 64, 42, 17, 5), (128, 64, 42, 20, 4),
                                          (128, 64, 63, 3, 1), (256, 128, 85, 9, 2),
                                          (256, 128, 127, 5, 3)])
def test_longitude_synthesis_against_fp64_sums(torch, I, J, N, K, nmem):
    """k_idft, a chunk of rows per block and whole columns, against FP64
    transforms of the same coefficients.  Bound per value: 2 M + 16 operations
    on terms that sum to the row's magnitudes."""
    stp = _grid_stepper(torch, I, J, N, K, nmem, "fp32")
    u, M = 2.0 ** -24, stp.M
    _noise(torch, stp.sf, 1)
    _noise(torch, stp.sfs, 2)
    stp.grid6.zero_()
    _launch(torch, stp, 4)
    rcos = stp.jfac.double().reshape(4, J)[2][None, :, None, None]
    S = stp.sfs.to(torch.complex128).permute(0, 2, 3, 1)       # [E][J][5][M]
    F = stp.sf.to(torch.complex128).permute(0, 2, 3, 4, 1)     # [E][J][K][6][M]
    m = torch.arange(M, device="cuda", dtype=torch.float64)
    rows = [S[:, :, :1], 1j * m * S[:, :, :1] * rcos, S[:, :, 1:4] * rcos, S[:, :, 4:5]]
    # surface fields: pi, H pi (pi_y), U-, V-, D-sum
    lev = F.clone()
    lev[:, :, :, :2] *= rcos[..., None]
    X = torch.cat(rows + [lev.reshape(nmem, J, 6 * K, M)], 2)
    want = torch.fft.irfft(X, n=I, dim=-1) * I
    two = torch.full((M,), 2.0, device="cuda", dtype=torch.float64)
    two[0] = 1.0
    size = (X.abs() * two).sum(-1, keepdim=True)
    err = (stp.grid6.double() - want).abs()
    assert bool((err <= (2 * M + 16) * u * size).all()), float((err / size).max() / u)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_forcings_set_in_turn_equal_fresh_ones(torch, precision):
    """A stepper whose forcings change (fields added, dropped, shared by the
    members, not contiguous, real) holds what a new stepper is given: the same values."""
    K, E = 5, 3
    one = _grid_stepper(torch, 64, 32, 21, K, E, precision)
    M = one.M
    g = torch.Generator().manual_seed(2)
    f = lambda *s: torch.randn(s, generator=g, dtype=torch.float64).cuda()      # noqa: E731
    c = lambda *s: torch.complex(f(*s), f(*s))                                  # noqa: E731
    for kw in (dict(frc_t=c(E, M, M, K)), dict(frc_t=c(M, M, K), frc_pi=c(E, M, M)),
               dict(frc_vor=c(E, M, M, K)), dict(frc_q=c(E, M, K, M).transpose(-1, -2)),
               dict(frc_div=f(1, M, M, K), frc_pi=c(1, M, M).cpu())):
        one.set_forcing(per_member=True, **kw)
        fresh = _grid_stepper(torch, 64, 32, 21, K, E, precision)
        fresh.set_forcing(per_member=True, **kw)
        torch.cuda.synchronize()
        assert torch.equal(one.frc3, fresh.frc3) and torch.equal(one.frcs, fresh.frcs)
        for i, n in enumerate(("vor", "div", "t", "q")):
            want = kw.get("frc_" + n)
            if want is None:
                assert not bool(one.frc3[:, i].any())
            else:
                want = want.reshape(-1, M, M, K)[:, one.pm, one.pn].to(one.cd)
                assert torch.equal(one.frc3[:, i], want.expand(E, -1, -1))
        if kw.get("frc_pi") is None:
            assert not bool(one.frcs.any())
        else:
            want = kw["frc_pi"].cuda()[..., one.pm, one.pn].reshape(-1, one.NS).to(one.cd)
            assert torch.equal(one.frcs, want.expand(E, -1))


@pytest.mark.parametrize("K,nmem", [(8, 1), (20, 3), (20, 75)])
def test_surface_rows_of_few_and_many_members(torch, K, nmem):
    """k_fdft_surf with two members a block against eight: the same bits for a
    member, and FP64 transforms within I + 16 roundings of the row's magnitudes."""
    few = _grid_stepper(torch, 64, 32, 21, K, nmem, "bf16x3")
    many = _grid_stepper(torch, 64, 32, 21, K, 83, "bf16x3")
    assert few.legendre and few.tc_dft is not None
    g = torch.Generator(device="cuda").manual_seed(K)
    few.grid9.copy_(torch.randn(few.grid9.shape, generator=g, device="cuda"))
    many.grid9.zero_()
    many.grid9[-nmem:].copy_(few.grid9)
    for s in (few, many):
        s.afs.zero_()
        _launch(torch, s, 6)
    assert torch.equal(few.afs, many.afs[-nmem:])
    x = few.grid9[:, :, :2].double()
    wg = few.jfac.double().reshape(4, 32)[0][None, :, None, None] / 64
    want = wg * torch.fft.rfft(x, dim=-1)[..., :few.M]
    got = few.afs.to(torch.complex128).permute(0, 2, 3, 1)
    size = wg * x.abs().sum(-1, keepdim=True)
    assert bool(((got - want).abs() <= (64 + 16) * 2.0 ** -24 * 2 * size).all())
