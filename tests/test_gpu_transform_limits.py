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


@pytest.mark.parametrize("J,N,C", [(2, 20, 349_600), (64, 1, 524_400)])
def test_more_columns_than_one_grid(torch, J, N, C):
    """Columns whose chunks and value parts exceed one grid's third dimension
    (analysis of the first shape, synthesis of the second): any slice of the
    columns equals a call on that slice, the same sums in the same order."""
    import lbm_isca_gb300.ops      # noqa: F401  (registers the operators)
    g = torch.Generator(device="cuda").manual_seed(J)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")     # noqa: E731
    M = N + 1
    t = rnd(M, M, J)
    fa, sa = (torch.view_as_complex(rnd(1, M, n, C, 2)) for n in (J, M))
    anal = lambda x: torch.ops.lbm_gb300.legendre_analysis(         # noqa: E731
        x, t, 0, None, None, 0, 0.0, None)
    synth = lambda x: torch.ops.lbm_gb300.legendre_synthesis(       # noqa: E731
        x, t, 0, None, None, None, 0, None, 0.0)
    for op, x in ((anal, fa), (synth, sa)):
        got = op(x)
        assert bool((got.abs().sum((0, 1, 2)) > 0).all())
        for c in (0, C // 2, C - 1000):
            assert torch.equal(got[..., c:c + 1000], op(x[..., c:c + 1000].contiguous()))
