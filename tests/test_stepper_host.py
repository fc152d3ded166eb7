"""Host side of the ensemble stepper on CPU tensors: packing of rectangles,
forcings, the grid-row workspace."""

import contextlib
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.fixture
def host_stepper(monkeypatch):
    """Makes EnsembleStepper objects that hold what packing and forcing need, on
    the CPU, with torch's stream calls replaced by nothing."""
    from lbm_isca_gb300.stepper import EnsembleStepper
    null = types.SimpleNamespace(wait_stream=lambda other: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: null)
    monkeypatch.setattr(torch.cuda, "default_stream", lambda *a: null)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())

    def make(N, K, E):
        s = object.__new__(EnsembleStepper)
        s.dev, s.cd = torch.device("cpu"), torch.complex128
        s.M, s.K, s.E, s.NS = N + 1, K, E, (N + 1) * (N + 2) // 2
        s.pm, s.pn = torch.triu_indices(s.M, s.M)
        s.pmn = s.pm * s.M + s.pn
        s.stream, s.frc3, s.frcs, s._graphs, s._desc = null, None, None, {}, None
        return s
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, s: None)
    return make


def _spec(g, *shape):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, dtype=torch.float64))


def test_as_many_levels_as_wavenumbers(host_stepper):
    """K = nmax + 1: a field's level axis is not taken for n, in the state and
    in a forcing that is not contiguous."""
    N, K, E = 4, 5, 3
    s, g = host_stepper(N, K, E), torch.Generator().manual_seed(1)
    x, pi = _spec(g, E, s.M, s.M, K), _spec(g, E, s.M, s.M)
    want, want_pi = x[:, s.pm, s.pn, :], pi[:, s.pm, s.pn]
    turned = x.permute(3, 2, 1, 0).contiguous().permute(3, 2, 1, 0)
    assert torch.equal(s._gather(turned, True), want)
    assert torch.equal(s._gather(x, True), want) and torch.equal(s._gather(pi, False), want_pi)
    assert torch.equal(s.pack(pi), want_pi)

    s.I = s.J = 2
    s.sa3 = torch.zeros((E, 4, s.NS, K), dtype=s.cd)
    s.sb3, s.sas = torch.zeros_like(s.sa3), torch.zeros((E, 4, s.NS), dtype=s.cd)
    s.psa = s.psb = torch.zeros((E, 2, 2), dtype=torch.float64)
    s.err, s.err_member = torch.zeros(1), torch.zeros(E)
    s.op_args = lambda: ()
    ops = types.SimpleNamespace(stepper_colsum=lambda: None, stepper_prime=lambda: None)
    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(torch.ops, "lbm_gb300", ops, raising=False)
        s.load({k: x for k in ("vor", "div", "t", "q")} | {"pi": pi},
               {k: x for k in ("vor", "div", "t", "q")}, s.psa, s.psb)
    for f in range(4):
        assert torch.equal(s.sa3[:, f], want) and torch.equal(s.sb3[:, f], want)
    assert torch.equal(s.sas[:, 0], want_pi)


@pytest.mark.parametrize("bad", [dict(frc_t=(3, True)), dict(frc_pi=(3, False)),
                                 dict(frc_vor=(2, True), frc_q=(3, True))])
def test_refused_forcing_leaves_the_old_one(host_stepper, bad):
    """A call with a field of a wrong number of members raises and changes
    nothing: neither the forcing in force nor what later calls leave."""
    N, K, E = 4, 3, 2
    s, g = host_stepper(N, K, E), torch.Generator().manual_seed(2)
    first = _spec(g, E, s.M, s.M, K)
    s.set_forcing(frc_t=first, per_member=True)
    f3, fs = s.frc3.clone(), s.frcs.clone()
    fields = dict(frc_vor=_spec(g, E, s.M, s.M, K), frc_pi=_spec(g, E, s.M, s.M))
    fields.update({k: _spec(g, n, s.M, s.M, *([K] if has_k else [])) for k, (n, has_k) in
                   bad.items()})
    with pytest.raises(RuntimeError):
        s.set_forcing(per_member=True, **fields)
    assert torch.equal(s.frc3, f3) and torch.equal(s.frcs, fs)
    s.set_forcing(frc_t=first, per_member=True)
    assert torch.equal(s.frc3, f3) and torch.equal(s.frcs, fs)


def test_replaced_buffers_outlive_the_queued_steps(host_stepper, monkeypatch):
    """Forcing and operator buffers belong to the caller's stream, queued steps
    read them on the stepper's: each set is recorded there before it is dropped."""
    N, K, E = 4, 3, 2
    s, g = host_stepper(N, K, E), torch.Generator().manual_seed(3)
    kept = []
    monkeypatch.setattr(torch.Tensor, "record_stream",
                        lambda t, st: kept.append((t.data_ptr(), id(st))))
    shared, per = _spec(g, s.M, s.M, K), _spec(g, E, s.M, s.M, K)
    s.set_forcing(frc_t=shared)
    for change in (lambda: s.set_forcing(frc_t=per, per_member=True), s.set_forcing):
        old = [t.data_ptr() for t in (s.frc3, s.frcs)]
        change()
        assert {(p, id(s.stream)) for p in old} <= set(kept)

    one = torch.eye(K, dtype=torch.float64)
    s.rd, s._dts, s.minv, s.vdm = torch.float64, [], None, None
    s.semi = types.SimpleNamespace(matrices=lambda dt: (None, one.expand(s.M, K, K), None))
    s.vdiff = types.SimpleNamespace(operators=lambda dt: dict.fromkeys(("vor", "div", "t", "q")))
    s.set_timesteps([600.0])
    old = [t.data_ptr() for t in (s.minv, s.vdm)]
    s.set_timesteps([1200.0])
    assert {(p, id(s.stream)) for p in old} <= set(kept)


@pytest.mark.parametrize("full", [(6 + 6 * 3,), (2 + 9 * 3,)])
def test_fp64_without_room_for_grid_rows(host_stepper, monkeypatch, full):
    """An FP64 stepper runs without the optional grid rows where the device has
    no memory left for them, or they exceed the limit; FP32 needs them."""
    s = host_stepper(4, 3, 2)
    s.J, s.I, s.precision, s.rd = 6, 16, "fp64", torch.float64
    assert [tuple(x.shape) for x in s._grid_rows()] == [(2, 6, 24, 16), (2, 6, 29, 16)]
    s.GRID_ROWS_BYTES = 8 * 2 * 6 * 53 * 16 - 1
    assert s._grid_rows() == (None, None)
    del s.GRID_ROWS_BYTES
    zeros = torch.zeros

    def no_room(shape, **kw):
        if shape[2] in full:
            raise torch.cuda.OutOfMemoryError("no room")
        return zeros(shape, **kw)
    monkeypatch.setattr(torch, "zeros", no_room)
    assert s._grid_rows() == (None, None)
    s.precision, s.rd = "fp32", torch.float32
    with pytest.raises(torch.cuda.OutOfMemoryError):
        s._grid_rows()
