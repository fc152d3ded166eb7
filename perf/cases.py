"""Performance cases: the work a program has this package do, through its
public entry points.

Kinds of a case:

* ``steps``: ``EnsembleStepper.run`` advances a loaded ensemble (what
  ``LBM.run`` does between two output days); the updated state comes back.
* ``forced``: a new steady forcing and one step, the loop of a time-varying
  forcing (one ``set_forcing`` and one step per call, no graph).
* ``run``: a whole ``LBM.run`` from rest with per-member heatings.
* ``transforms``: ``Spectral`` scalar and wind transforms, both directions.
* ``gradient``: ``ForcingGradient.value_and_grad`` (forward sweep and adjoint).

Grids, level counts, member counts, precisions and model settings are those of
the package's configurations, tests and benchmark.  The basic state is
``configs.solid_body_basic_state`` with a humidity profile, so that the
moisture terms work on non-zero fields.

``exact`` restates the model in plain float64 torch: Gauss-Legendre grid,
Legendre recurrences, Simmons-Burridge levels, linearised primitive equations,
semi-implicit leapfrog with Robert-Asselin filter.
"""

import math
import types

import numpy as np
import torch

GRIDS = {"T21": (64, 32, 21), "T42": (128, 64, 42), "T85": (256, 128, 85)}
DELT = {"T21": 1200.0, "T42": 1200.0, "T85": 600.0}
FIELDS = ("vor", "div", "t", "q")


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _case(name, kind, grid, levels, members, precision, steps, config="plain"):
    c = {"kind": kind, "grid": grid, "levels": levels, "members": members,
         "precision": precision, "steps": steps, "config": config}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one member under a time-varying forcing: a new forcing field and one
        # step per call; launches and host work count
        _case("forced_step_t21l20_m1_fp32", "forced", "T21", 20, 1, "fp32", 1),
        # the default model, one member in FP64, over one model day
        _case("day_t42l20_m1_fp64", "steps", "T42", 20, 1, "fp64", 72, "default"),
        # the same in single precision
        _case("day_t42l20_m1_fp32", "steps", "T42", 20, 1, "fp32", 72, "default"),
        # a handful of members on an odd number of levels
        _case("steps_t42l17_m7_fp32", "steps", "T42", 17, 7, "fp32", 12),
        # the low-resolution group of a mixed ensemble, two-way bf16 split
        _case("steps_t21l20_m48_bf16split", "steps", "T21", 20, 48, "bf16split", 12),
        # the ensemble of the precision sweep
        _case("steps_t42l20_m128_fp32", "steps", "T42", 20, 128, "fp32", 4),
        # the benchmark ensemble
        _case("steps_t42l20_m512_bf16x3", "steps", "T42", 20, 512, "bf16x3", 4),
        # the high-resolution group of a mixed ensemble
        _case("steps_t85l40_m16_bf16x3", "steps", "T85", 40, 16, "bf16x3", 4),
        # a reference-precision ensemble
        _case("steps_t42l20_m32_fp64", "steps", "T42", 20, 32, "fp64", 2),
        # analysis and synthesis of an ensemble's winds and temperature
        _case("transforms_t42l20_m32_fp64", "transforms", "T42", 20, 32, "fp64", 1),
        # sensitivity of a response to the heating: forward and adjoint
        _case("gradient_t42l20_m1_fp64", "gradient", "T42", 20, 1, "fp64", 6),
        # a whole call from rest: heatings in, half a day, grid fields out
        _case("run_t42l20_m8_bf16x3", "run", "T42", 20, 8, "bf16x3", 36),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(("steps", "steps", "steps", "steps", "forced", "run", "transforms",
                       "gradient"))
    grid = rng.choice(("T21", "T42", "T42", "T85"))
    if kind == "transforms":
        most = {"T21": 256, "T42": 64, "T85": 12}[grid]
        return _case(None, kind, grid, rng.randint(7, 40), log(1, most),
                     rng.choice(("fp64", "fp32")), 1)
    if kind == "gradient":
        grid = rng.choice(("T21", "T42"))
        return _case(None, kind, grid, rng.randint(8, 24), log(1, 4),
                     rng.choice(("fp64", "fp32")), rng.randint(2, 6))
    precision = rng.choice(("fp64", "fp32", "fp32", "bf16x3", "bf16x3", "bf16split"))
    if kind == "forced":
        grid = rng.choice(("T21", "T42"))
        levels = rng.randint(8, 28)
    else:
        levels = rng.randint(10, 40)
    if precision.startswith("bf16"):
        # even level counts that the tensor-core plans of the grid take
        lo, hi = {"T21": (4, 14), "T42": (4, 10), "T85": (17, 20)}[grid]
        levels = 2 * rng.randint(lo, hi)
    if kind == "forced":
        return _case(None, kind, grid, levels, log(1, 4), precision, 1)
    most = {"T21": 512, "T42": 256, "T85": 24}[grid]
    if precision == "fp64":
        most = max(1, most // 24)
    if kind == "run":
        return _case(None, kind, grid, levels, log(1, max(1, most // 16)), precision,
                     rng.randint(3, 24))
    members = log(1, most)
    return _case(None, kind, grid, levels, members, precision,
                 rng.randint(2, 4) if members > most // 16 else log(2, 24))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _sigma(case):
    from lbm_isca_gb300 import configs, constants
    if case["config"] == "default":
        return np.array(constants.SIGM)
    return configs.equal_sigma_half_levels(case["levels"])


def _config_values(case):
    """Model settings: the package's default settings, or the benchmark's plain damping."""
    from lbm_isca_gb300 import configs
    delt = DELT[case["grid"]]
    if case["config"] == "default":
        return {"delt": delt}
    return dict(configs.plain_damping(case["levels"]), delt=delt)


def _basic_state(case):
    from lbm_isca_gb300 import configs
    I, J, _ = GRIDS[case["grid"]]
    sigm = _sigma(case)
    bs = configs.solid_body_basic_state(I, J, sigm)
    mu, _ = configs.gaussian_latitudes(J)
    sig = configs.full_level_sigma(sigm)
    bs.q = np.broadcast_to(0.014 * (1.0 - mu * mu)[:, None, None] * (sig ** 3)[None, None, :],
                           bs.t.shape).copy()
    return bs


def _random_spectrum(gen, members, nmax, sig, amp, n0=8.0, slope=1.5):
    """Random coefficients (members, m, n, k) of a smooth field with RMS of
    order amp, red in n, a few vertical modes deep, m = 0 real, representable
    in float32; (members, m, n) for sig None."""
    M = nmax + 1
    dev = gen.device
    n = torch.arange(M, device=dev, dtype=torch.float64)
    shape = (n0 / (n + n0)) ** slope * (n > 0)
    mask = torch.triu(torch.ones((M, M), device=dev, dtype=torch.float64)) * shape
    mask = mask / (mask.square().sum() ** 0.5)
    nz = 1 if sig is None else 4
    x = torch.randn((members, M, M, nz, 2), generator=gen, device=dev, dtype=torch.float32)
    x = x.to(torch.float64) * (amp * mask)[None, :, :, None, None]
    x[:, 0, :, :, 1] = 0.0
    if sig is None:
        x = x[:, :, :, 0]
    else:
        l = torch.arange(nz, device=dev, dtype=torch.float64)
        s = torch.as_tensor(sig, device=dev)
        modes = torch.cos(math.pi * l[:, None] * s[None, :]) / (1.0 + l[:, None])
        x = torch.einsum("emnlc,lk->emnkc", x, modes)
    return torch.view_as_complex(x.float().double().contiguous())


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _spectral_state(case, seed):
    """Two time levels of an ensemble: a (vor, div, t, q, pi), b (vor, div, t,
    q), grid ps of both, and per-member heating; all float32 values in float64."""
    from lbm_isca_gb300 import configs
    I, J, N = GRIDS[case["grid"]]
    E = case["members"]
    g = _generator(seed)
    sig = configs.full_level_sigma(_sigma(case))
    amp = {"vor": 8e-6, "div": 4e-7, "t": 0.8, "q": 1.5e-4}
    a = {k: _random_spectrum(g, E, N, sig, amp[k]) for k in FIELDS}
    a["pi"] = _random_spectrum(g, E, N, None, 4e-4)
    b = {k: (a[k] + _random_spectrum(g, E, N, sig, 0.02 * amp[k])).to(torch.complex64)
         .to(torch.complex128) for k in FIELDS}
    lat = torch.rand((E, 8, 1, 1), generator=g, device="cuda", dtype=torch.float64)
    y = torch.linspace(-1.0, 1.0, J, device="cuda", dtype=torch.float64)[None, :, None]
    x = torch.arange(I, device="cuda", dtype=torch.float64)[None, None, :] * (2.0 * math.pi / I)

    def ps(i):
        p = 0.4 * torch.cos(2.0 * x + 6.0 * lat[:, i]) * (1.0 - y * y)
        p = p + 0.2 * torch.sin(3.0 * x + 6.0 * lat[:, i + 1]) * y * (1.0 - y * y)
        return p.float().double()

    psa = ps(0)
    psb = (psa + 0.02 * ps(2)).float().double()
    return a, b, psa, psb, _heating_spectrum(case, g)


def _heating_spectrum(case, g):
    from lbm_isca_gb300 import configs
    sig = configs.full_level_sigma(_sigma(case))
    return _random_spectrum(g, case["members"], GRIDS[case["grid"]][2], sig, 1.0 / 86400.0, n0=5.0)


def _grid_heating(case, seed):
    """Compact heatings on the grid, one per member (K/s)."""
    from lbm_isca_gb300 import configs
    I, J, _ = GRIDS[case["grid"]]
    h, _ = configs.ensemble_heating(I, J, _sigma(case), case["members"], int(seed))
    return h


def _model(case):
    from lbm_isca_gb300 import LBM, BatchedSpectral, Config, Spectral, VerticalGrid
    I, J, N = GRIDS[case["grid"]]
    precision = "fp64" if case["kind"] == "gradient" else case["precision"]
    cfg = Config(precision=precision, nmem=case["members"],
                 ndays=case["steps"] * DELT[case["grid"]] / 86400.0, **_config_values(case))
    plain = Spectral(nlon=I, nlat=J, nmax=N)
    batched = BatchedSpectral(nlon=I, nlat=J, nmax=N) if case["members"] > 1 else plain
    return LBM(_basic_state(case), batched, VerticalGrid(sigm=_sigma(case)), cfg,
               basic_spectral=plain)


def prepare(case, seed):
    s = types.SimpleNamespace(kind=case["kind"])
    if case["kind"] == "transforms":
        from lbm_isca_gb300 import BatchedSpectral
        I, J, N = GRIDS[case["grid"]]
        s.sp = BatchedSpectral(nlon=I, nlat=J, nmax=N, precision=case["precision"])
        s.u, s.v, s.t = _wind_inputs(case, seed)
        return s
    s.model = _model(case)
    s.dt = DELT[case["grid"]]
    if case["kind"] in ("steps", "forced"):
        a, b, psa, psb, heat = _spectral_state(case, seed)
        s.stepper = s.model.stepper()
        s.stepper.set_timesteps([s.dt])
        s.stepper.set_forcing(frc_t=heat, per_member=True)
        s.stepper.load(a, b, psa, psb)
        s.calls = [(s.dt, False)] * case["steps"]
        if case["kind"] == "forced":
            s.heat = heat
    elif case["kind"] == "run":
        s.heat = torch.as_tensor(_grid_heating(case, seed)).cuda()
        if case["members"] == 1:
            s.heat = s.heat[0]
        s.forcing = types.SimpleNamespace(vor=None, div=None, t=s.heat, ps=None)
        s.rest = torch.zeros_like(s.heat)
    else:
        from lbm_isca_gb300.adjoint import AreaMeanStreamfunction, ForcingGradient
        s.heat = torch.as_tensor(_grid_heating(case, seed)).cuda()
        if case["members"] == 1:
            s.heat = s.heat[0]
        s.gradient = ForcingGradient(s.model, AreaMeanStreamfunction(s.model.sp, s.model.vg),
                                     nsteps=case["steps"], precision=case["precision"])
        if case["precision"] == "fp32":
            # the response in the working precision of the sweep
            s.gradient.response = AreaMeanStreamfunction(s.gradient.step.sp, s.model.vg)
    return s


def _wind_inputs(case, seed):
    """Grid winds and temperature with noise at every scale, float32 values."""
    I, J, _ = GRIDS[case["grid"]]
    g = _generator(seed)
    shape = (case["members"], J, I, case["levels"])
    y = torch.linspace(-1.0, 1.0, J, device="cuda", dtype=torch.float64)[None, :, None, None]
    rd = torch.float64 if case["precision"] == "fp64" else torch.float32

    def field(amp):
        r = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
        return (amp * (1.0 - y * y) * r).float().to(rd)

    return field(8.0), field(5.0), field(2.0)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _stepper_outputs(stp):
    # the caller's stream reads the state once the stepper's stream has written it
    torch.cuda.current_stream().wait_stream(stp.stream)
    a, b = stp.sa3.unbind(1), stp.sb3.unbind(1)
    return {"vor": a[0], "div": a[1], "t": a[2], "q": a[3], "pi": stp.sas[:, 0],
            "vor_b": b[0], "div_b": b[1], "t_b": b[2], "q_b": b[3],
            "ps_a": stp.psa, "ps_b": stp.psb}


def run(s):
    if s.kind == "steps":
        s.stepper.run(s.calls)
        return _stepper_outputs(s.stepper)
    if s.kind == "forced":
        s.stepper.set_forcing(frc_t=s.heat, per_member=True)
        s.stepper.run(s.calls, use_graph=False)
        return _stepper_outputs(s.stepper)
    if s.kind == "run":
        m = s.model
        m.set_initial_perturbation(u=s.rest, v=s.rest, t=s.rest, q=s.rest, ps=s.rest[..., 0])
        m.time = 0.0
        m.run(steady_forcing=s.forcing, verbose=False)
        return {x + n: getattr(st, n) for x, st in (("a_", m.ga), ("b_", m.gb))
                for n in ("u", "v", "t", "q", "ps")}
    if s.kind == "transforms":
        vor, div = s.sp.uv_to_vordiv(s.u, s.v)
        u, v = s.sp.vordiv_to_uv(vor, div)
        t = s.sp.grid_to_wave(s.t)
        return {"vor": vor, "div": div, "t": t, "u_grid": u, "v_grid": v,
                "t_grid": s.sp.wave_to_grid(t)}
    value, grad = s.gradient.value_and_grad(s.heat)
    return {"value": value, "grad": grad}


# ---------------------------------------------------------------------------
# Work of one pass
# ---------------------------------------------------------------------------
def work(case):
    I, J, N = GRIDS[case["grid"]]
    M, K, E = N + 1, case["levels"], case["members"]
    NS = M * (M + 1) // 2
    w = 8 if case["precision"] == "fp64" else 4
    fft = 2.5 * I * math.log2(I)                       # one real row
    leg = 4.0 * NS * (J // 2)                          # one complex column, parity used
    grid, spec = J * I * K * w, 2 * M * M * K * w
    if case["kind"] == "transforms":
        return {"bytes": E * (6 * grid + 3 * spec),
                "flops": E * K * (6 * J * fft + 10 * leg)}
    state = 2 * w * NS * (8 * K + 1) + 2 * w * J * I
    basic = w * J * I * (15 * K + 6) + 2 * w * NS * J
    flops = E * ((15 * K + 8) * J * fft + (17 * K + 9) * leg + 200.0 * J * I * K
                 + NS * K * (8.0 * K + 100.0))
    calls = case["steps"]
    if case["kind"] == "forced":
        return {"bytes": E * (2 * state + 2 * 2 * w * NS * K) + basic, "flops": flops}
    if case["kind"] == "steps":
        return {"bytes": calls * E * 2 * state + basic + E * 2 * w * NS * K,
                "flops": calls * flops}
    calls += 2                                         # the start-up calls
    if case["kind"] == "run":
        return {"bytes": E * (calls * 2 * state + 8 * J * I * (9 * K + 2)) + basic,
                "flops": calls * flops}
    # gradient: every call forward once, and its adjoint
    return {"bytes": E * (calls * 4 * state + 2 * grid) + 2 * basic, "flops": 2.5 * calls * flops}


# ---------------------------------------------------------------------------
# The same in plain float64
# ---------------------------------------------------------------------------
ER, OMEGA, RAIR, KAPPA = 6.371e6, 7.2921150e-5, 287.04, 2.0 / 7.0
EPSVT = 461.50 / 287.04 - 1.0
DAY = 86400.0
# default model settings: drag times in days, hyperdiffusion, sponge, diffusion
DRAG = [0.5, 0.5, 0.5, 5, 15, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 20, 0.5, 0.5]


class _Sphere:
    """Spherical-harmonic transforms on (batch, lat, lon, column) arrays."""

    def __init__(self, I, J, N):
        self.I, self.J, self.M = I, J, N + 1
        M = N + 1
        x, w = np.polynomial.legendre.leggauss(J)
        mu, gw = x[::-1].copy(), w[::-1].copy() / 2.0
        cos = np.sqrt(1.0 - mu * mu)
        eps = np.zeros((M, N + 2))
        for m in range(M):
            k = np.arange(m + 1, N + 2, dtype=np.float64)
            eps[m, m + 1:] = np.sqrt((k * k - m * m) / (4.0 * k * k - 1.0))
        P = np.zeros((M, N + 2, J))
        H = np.zeros((M, M, J))
        top = np.ones(J)
        for m in range(M):
            if m:
                top = top * math.sqrt((2.0 * m + 1.0) / (2.0 * m)) * cos
            P[m, m] = top
            P[m, m + 1] = top * math.sqrt(2.0 * m + 3.0) * mu
            for k in range(m + 2, N + 2):
                P[m, k] = (mu * P[m, k - 1] - eps[m, k - 1] * P[m, k - 2]) / eps[m, k]
            for k in range(m, M):
                H[m, k] = -k * eps[m, k + 1] * P[m, k + 1]
                if k > m:
                    H[m, k] += (k + 1.0) * eps[m, k] * P[m, k - 1]
        T = lambda a: torch.as_tensor(a, device="cuda")       # noqa: E731
        self.mu, self.gw = mu, gw
        self.P, self.H = T(P[:, :M].copy()), T(H)
        gd = gw / ER / (1.0 - mu * mu)
        self.Pg, self.Pd, self.Hd = self.P * T(gw), self.P * T(gd), self.H * T(gd)
        self.cos = T(cos)[:, None, None]
        n = torch.arange(M, device="cuda", dtype=torch.float64)
        self.lap = -n * (n + 1.0) / ER ** 2
        self.invlap = torch.where(n > 0, -ER ** 2 / (n * (n + 1.0)).clamp(min=1.0), 0.0)
        self.im = (1j * n)[:, None, None]

    def fwd(self, g):
        """(B, J, I, C) -> (B, M, J, C)"""
        return (torch.fft.rfft(g, dim=2) / self.I)[:, :, :self.M].transpose(1, 2)

    def inv(self, F):
        F = torch.cat([F[:, :1].real.to(F.dtype), F[:, 1:]], 1).transpose(1, 2)
        return torch.fft.irfft(F * self.I, n=self.I, dim=2)

    def _mul(self, eq, table, x):
        return torch.view_as_complex(torch.einsum(eq, table, torch.view_as_real(x.contiguous()))
                                     .contiguous())

    def anal(self, F, table):
        return self._mul("mnj,bmjcr->bmncr", table, F)

    def synth(self, S, table):
        return self._mul("mnj,bmncr->bmjcr", table, S)

    def to_wave(self, g):
        return self.anal(self.fwd(g), self.Pg)

    def to_grid(self, S):
        return self.inv(self.synth(S, self.P))

    def vordiv(self, u, v):
        U, V = self.fwd(u * self.cos), self.fwd(v * self.cos)
        return (self.anal(self.im * V, self.Pd) + self.anal(U, self.Hd),
                self.anal(self.im * U, self.Pd) - self.anal(V, self.Hd))

    def wind(self, vor, div):
        psi, chi = vor * self.invlap[:, None], div * self.invlap[:, None]
        r = 1.0 / (ER * self.cos)
        return (self.inv(self.im * self.synth(chi, self.P) - self.synth(psi, self.H)) * r,
                self.inv(self.im * self.synth(psi, self.P) + self.synth(chi, self.H)) * r)

    def grad(self, S):
        r = 1.0 / (ER * self.cos)
        return (self.inv(self.im * self.synth(S, self.P)) * r,
                self.inv(self.synth(S, self.H)) * r)


def _seconds(days, K):
    """1 / (drag time) per level; none where the time is not positive."""
    out = np.zeros(K)
    if days is not None:
        d = np.asarray(days, dtype=np.float64) * DAY
        out[d > 0] = 1.0 / d[d > 0]
    return out


class _Model:
    """Linearised primitive equations with a semi-implicit leapfrog step."""

    def __init__(self, case):
        I, J, N = GRIDS[case["grid"]]
        K = case["levels"]
        self.K = K
        self.sp = sp = _Sphere(I, J, N)
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")    # noqa: E731
        h = _sigma(case)
        bot, top = h[:-1], h[1:]
        ds = bot - top
        safe = np.where(top > 0.0, top, 1.0)
        lr = np.where(top > 0.0, np.log(bot) - np.log(safe), 0.0)
        alpha = 1.0 - np.where(top > 0.0, top * lr / ds, 0.0)
        sig = bot * np.exp(-alpha)
        self.sig = sig
        d2 = np.where(top > 0.0, np.log(sig) - np.log(safe), 0.0)
        cpg = (bot * alpha + top * d2) / ds
        w3 = lr / ds
        ww = np.tril(np.ones((K, K)), -1) * (RAIR * lr)[None, :] + np.diag(RAIR * alpha)
        bs = _basic_state(case)
        g = lambda a: T(a)[None]                                # noqa: E731
        self.u, self.v, self.t, self.q = g(bs.u), g(bs.v), g(bs.t), g(bs.q)
        self.ps = g(bs.ps)
        self.tv = self.t * (1.0 + EPSVT * self.q)
        tref = self.tv.mean((0, 1, 2)).cpu().numpy()
        tm = KAPPA * tref[:, None] * w3[:, None] * np.triu(np.ones((K, K)), 1) * ds[None, :]
        tm = tm + np.diag(KAPPA * tref * alpha)
        gg = RAIR * tref * cpg
        self.ds, self.h, self.alpha, self.w3, self.wP = T(ds), T(h), T(alpha), T(w3), T(alpha - cpg)
        self.ww, self.tm, self.gg, self.rcpg = T(ww), T(tm), T(gg), T(RAIR * cpg)
        self.tref = T(tref)
        vor, div = sp.vordiv(self.u, self.v)
        self.div = sp.to_grid(div)
        self.absvor = sp.to_grid(vor) + 2.0 * OMEGA * T(sp.mu)[:, None, None]
        px, py = sp.grad(sp.to_wave(torch.log(self.ps)[..., None]))
        self.px, self.py = px, py                               # (1, J, I, 1)
        padv = self.u * px + self.v * py
        S = self.colsum(self.div + padv)
        self.sdot = self.sigmadot(S)
        self.x5 = self.w3 * S[..., 1:] + self.alpha * self.div + self.wP * padv
        # damping rates (n, k)
        c = _config_values(case)
        n = np.arange(N + 1, dtype=np.float64)
        order, tau = c.get("hdif_order", 4), c.get("hdif_tefold", 2.0) * 3600.0
        p = order // 2
        top_ = (N + 1.0) ** p
        kt = (n * (n + 1.0) / N) ** p / top_ / tau
        kv = ((n * (n + 1.0) / N) ** p - (2.0 / N) ** p) / top_ / tau
        kt[0] = kv[0] = 0.0
        kv[1] = max(kv[1], 0.0)
        sponge = np.zeros(K)
        if c.get("sponge", True):
            z = -8.0e3 * np.log(sig)
            sponge = np.maximum(1.0 + np.tanh((z - z[-1]) / 7.0e3), 1e-20) / (30.0 * 3600.0)
        drag = {x: _seconds(c.get("ddrag" + x, None if x == "q" else DRAG), K) for x in "vdtq"}
        self.kv = T(kv[:, None] + (sponge + drag["v"])[None])
        self.kd = T(kv[:, None] + (sponge + drag["d"])[None])
        self.kt = T(kt[:, None] + drag["t"][None])
        self.kq = T(kt[:, None] + drag["q"][None])
        self.robert = c.get("robert", 0.04)
        self.linear = c.get("strictly_linear", False)
        # vertical diffusion: sigma-space Laplacian and coefficients
        dm = np.concatenate([[h[0] - sig[0]], sig[:-1] - sig[1:], [sig[-1] - h[-1]]])
        lop = np.zeros((K, K))
        for k in range(K):
            if k > 0:
                lop[k, k - 1] = 1.0 / (ds[k] * dm[k])
            if k < K - 1:
                lop[k, k + 1] = 1.0 / (ds[k] * dm[k + 1])
        lop[0, 1] = (dm[0] + dm[1]) / (ds[0] * dm[0] * dm[1])
        lop[K - 1, K - 2] = (dm[K - 1] + dm[K]) / (ds[K - 1] * dm[K - 1] * dm[K])
        lop -= np.diag(lop.sum(1))
        nu = {}
        for x, default in (("v", 1e3), ("d", 1e3), ("t", 1e3), ("q", None)):
            val = c.get("vdif" + x, default)
            nu[x] = None if val is None else 1.0 / (DAY * val)
        self.lop, self.nu = lop, nu
        self.cache = {}

    def operators(self, dt):
        if dt not in self.cache:
            K, lap = self.K, self.sp.lap
            eye = torch.eye(K, device="cuda", dtype=torch.float64)
            wh, gc = self.ww @ self.tm, torch.outer(self.gg, self.ds)
            ft, fd = 1.0 + 2.0 * dt * self.kt, 1.0 + 2.0 * dt * self.kd
            m = (ft * fd)[:, :, None] * eye - dt * dt * lap[:, None, None] * (
                wh[None] + ft[:, :, None] * gc[None])
            vd = {x: None if v is None else torch.linalg.inv(
                eye - dt * v * torch.as_tensor(self.lop, device="cuda"))
                for x, v in self.nu.items()}
            self.cache[dt] = (torch.linalg.inv(m), vd)
        return self.cache[dt]

    def colsum(self, x):
        w = torch.flip(torch.cumsum(torch.flip(x * self.ds, (-1,)), -1), (-1,))
        return torch.cat([w, torch.zeros_like(w[..., :1])], -1)

    def sigmadot(self, S):
        s = self.h * S[..., :1] - S
        return torch.cat([torch.zeros_like(s[..., :1]), s[..., 1:-1],
                          torch.zeros_like(s[..., :1])], -1)

    def vadv(self, f, s):
        mid = s[..., 1:-1] * 0.5 * (f[..., 1:] + f[..., :-1])
        z = torch.zeros_like(mid[..., :1])
        F = torch.cat([z, mid, z], -1)
        return (F[..., 1:] - F[..., :-1] - f * (s[..., 1:] - s[..., :-1])) / self.ds

    def tendencies(self, a, heat):
        """a: spectral state; heat: spectral heating; -> spectral tendencies."""
        sp = self.sp
        u, v = sp.wind(a["vor"], a["div"])
        vo, dv, t, q = (sp.to_grid(a[k]) for k in FIELDS)
        px, py = sp.grad(a["pi"][..., None])
        padv = u * self.px + self.u * px + v * self.py + self.v * py
        S = self.colsum(dv + padv)
        s, sb = self.sigmadot(S), self.sdot
        mix = EPSVT * (t * self.q + self.t * q)
        tv = t + mix
        tdev, tvdev = self.t - self.tref, self.tv - self.tref
        x5 = self.alpha * dv + self.wP * padv + self.w3 * S[..., 1:]
        gt = (-KAPPA * (tv * self.x5 + self.tv * x5) + t * self.div + tdev * dv
              + self.vadv(t, sb) + self.vadv(self.t.expand_as(t), s) + dv @ self.tm.T)
        fu = (v * self.absvor + self.v * vo - self.rcpg * (tv * self.px + tvdev * px)
              + self.vadv(u, sb) + self.vadv(self.u.expand_as(u), s))
        fv = (-u * self.absvor - self.u * vo - self.rcpg * (tv * self.py + tvdev * py)
              + self.vadv(v, sb) + self.vadv(self.v.expand_as(v), s))
        ke = mix @ self.ww.T + u * self.u + v * self.v
        if not self.linear:
            ke = ke + 0.5 * (u * u + v * v)
        gq = (q * self.div + self.q * dv + self.vadv(q, sb)
              + self.vadv(self.q.expand_as(q), s))
        wv, wd = sp.vordiv(fu, fv)
        wd = wd - sp.lap[:, None] * sp.to_wave(ke)
        wt = sp.to_wave(gt) - sp.vordiv(u * tdev + self.u * t, v * tdev + self.v * t)[1]
        wq = sp.to_wave(gq) - sp.vordiv(u * self.q + self.u * q, v * self.q + self.v * q)[1]
        wp = sp.to_wave(-(padv * self.ds).sum(-1, keepdim=True))[..., 0]
        return {"vor": wv, "div": wd, "t": wt if heat is None else wt + heat, "q": wq, "pi": wp}

    def implicit(self, dt, b, w):
        minv, vd = self.operators(dt)
        c = lambda m, x: torch.complex(x.real @ m, x.imag @ m)       # noqa: E731
        lap = self.sp.lap[:, None]
        ft = 1.0 + 2.0 * dt * self.kt
        wx = b["t"] * (1.0 + dt * self.kt) + dt * w["t"]
        wp = (b["pi"] + dt * w["pi"])[..., None]
        phi = c(self.ww.T, wx) + ft * self.gg * wp
        rhs = b["div"] * (1.0 + dt * self.kd) * ft + dt * (w["div"] * ft - lap * phi)
        dbar = torch.complex(torch.einsum("nkl,bmnl->bmnk", minv, rhs.real.contiguous()),
                             torch.einsum("nkl,bmnl->bmnk", minv, rhs.imag.contiguous()))
        new = {"vor": (b["vor"] + 2.0 * dt * w["vor"]) / (1.0 + 2.0 * dt * self.kv),
               "div": 2.0 * dbar - b["div"],
               "t": (b["t"] + 2.0 * dt * (w["t"] - c(self.tm.T, dbar))) / ft,
               "q": (b["q"] + 2.0 * dt * w["q"]) / (1.0 + 2.0 * dt * self.kq),
               "pi": b["pi"] + 2.0 * dt * (w["pi"] - (dbar * self.ds).sum(-1))}
        for name, x in zip(FIELDS, "vdtq"):
            if vd[x] is not None:
                y = c(vd[x].T, new[name])
                new[name] = (torch.cat([new[name][:, :, :2], y[:, :, 2:]], 2) if x in "vd" else y)
        return new

    def surface(self, a, psa, psb, mode):
        """Grid ps of the current and the filtered previous level."""
        now = self.ps * torch.expm1(self.sp.to_grid(a["pi"][..., None])[..., 0])
        if mode == 1:
            return now, psa
        if mode == 2:
            return now, psa + self.robert * (psb - 2.0 * psa + now)
        return psa, psb

    def advance(self, a, b, psa, psb, calls, heat, mode=0):
        """The calls [(dt, start)] from two spectral levels; mode: how ps of the
        previous level is brought up to date (0 as given, 1 copy, 2 filter)."""
        for dt, start in calls:
            psa, psb = self.surface(a, psa, psb, mode)
            w = self.tendencies(a, heat)
            prev = dict(b, pi=self.sp.to_wave(torch.log1p(psb / self.ps)[..., None])[..., 0])
            new = self.implicit(dt, prev, w)
            b = {k: a[k] if start else a[k] + self.robert * (b[k] - 2.0 * a[k] + new[k])
                 for k in FIELDS}
            a, mode = new, 1 if start else 2
        return a, b, psa, psb, mode


def _rest(case, members):
    I, J, N = GRIDS[case["grid"]]
    z = torch.zeros((members, N + 1, N + 1, case["levels"]), device="cuda", dtype=torch.complex128)
    p = torch.zeros((members, J, I), device="cuda", dtype=torch.float64)
    a = {k: z for k in FIELDS}
    return dict(a, pi=z[..., 0]), a, p, p


def _schedule(case):
    d = DELT[case["grid"]]
    return [(d / 4.0, True), (d / 2.0, True)] + [(d, False)] * case["steps"]


def _parts(case):
    """Members in blocks that fit the device with the temporaries of a step."""
    I, J, _ = GRIDS[case["grid"]]
    size = max(1, int(2.5e8 / (8.0 * I * J * case["levels"])))
    return [(i, min(i + size, case["members"])) for i in range(0, case["members"], size)]


def _joined(parts):
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}


def exact(case, seed):
    if case["kind"] == "transforms":
        sp = _Sphere(*GRIDS[case["grid"]])
        got = []
        u, v, t = (x.double() for x in _wind_inputs(case, seed))
        for i, j in _parts(case):
            vor, div = sp.vordiv(u[i:j], v[i:j])
            s = sp.to_wave(t[i:j])
            ug, vg = sp.wind(vor, div)
            got.append({"vor": vor, "div": div, "t": s, "u_grid": ug, "v_grid": vg,
                        "t_grid": sp.to_grid(s)})
        return _joined(got)
    model = _Model(case)
    sp = model.sp
    if case["kind"] in ("steps", "forced"):
        a, b, psa, psb, heat = _spectral_state(case, seed)
        calls = [(DELT[case["grid"]], False)] * case["steps"]
        m, n = np.nonzero(np.triu(np.ones((sp.M, sp.M), dtype=bool)))
        got = []
        for i, j in _parts(case):
            x, y, pa, pb, _ = model.advance({k: f[i:j] for k, f in a.items()},
                                            {k: f[i:j] for k, f in b.items()},
                                            psa[i:j], psb[i:j], calls, heat[i:j])
            part = {k: x[k][:, m, n] for k in FIELDS + ("pi",)}
            part.update({k + "_b": y[k][:, m, n] for k in FIELDS}, ps_a=pa, ps_b=pb)
            got.append(part)
        return _joined(got)
    heat = torch.as_tensor(_grid_heating(case, seed)).cuda()
    single = case["members"] == 1
    if case["kind"] == "run":
        got = []
        for i, j in _parts(case):
            a, b, psa, psb, mode = model.advance(*_rest(case, j - i), _schedule(case),
                                                 sp.to_wave(heat[i:j]))
            psa, psb = model.surface(a, psa, psb, mode)
            part = {}
            for x, s, ps in (("a_", a, psa), ("b_", b, psb)):
                part[x + "u"], part[x + "v"] = sp.wind(s["vor"], s["div"])
                part[x + "t"], part[x + "q"] = sp.to_grid(s["t"]), sp.to_grid(s["q"])
                part[x + "ps"] = ps
            got.append(part)
        out = _joined(got)
        return {k: x[0] for k, x in out.items()} if single else out
    # gradient of the area-mean streamfunction by reverse differentiation
    with torch.enable_grad():
        h = heat.clone().requires_grad_(True)
        a = model.advance(*_rest(case, case["members"]), _schedule(case), sp.to_wave(h))[0]
        k = int(np.argmin(np.abs(model.sig - 0.25)))
        psi = sp.to_grid((a["vor"] * sp.invlap[:, None])[..., k:k + 1])[..., 0]
        lat, lon = np.degrees(np.arcsin(sp.mu)), np.arange(sp.I) * 360.0 / sp.I
        box = ((lat >= 30.0) & (lat <= 60.0))[:, None] & ((lon >= 150.0) & (lon <= 210.0))[None]
        wgt = box * sp.gw[:, None]
        value = (psi * torch.as_tensor(wgt / wgt.sum(), device="cuda")).sum((1, 2))
        (grad,) = torch.autograd.grad(value.sum(), h)
    value = value.detach()
    return {"value": value[0], "grad": grad[0]} if single else {"value": value, "grad": grad}
