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


@pytest.mark.parametrize("J,N,C,dtype", [(2, 20, 349_600, "float64"),
                                         (64, 1, 1_048_600, "float32")])
def test_more_columns_than_one_grid(torch, J, N, C, dtype):
    """Columns whose chunks and value parts exceed one grid's third dimension
    (analysis of the first shape, synthesis of the second): any slice of the
    columns equals a call on that slice, the same sums in the same order."""
    import lbm_isca_gb300.ops      # noqa: F401  (registers the operators)
    rt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(J)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=rt)     # noqa: E731
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


@pytest.mark.parametrize("B,J,N,C", [(40, 64, 42, 48), (12, 64, 42, 25), (20, 50, 31, 16),
                                     (64, 32, 21, 31), (10, 6, 3, 96)])
@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_batches_that_fill_sixteen_column_chunks(torch, B, J, N, C, two, dtype):
    """The form that stages whole sums, full chunks and ones with idle lanes: the
    bounds of the flat form."""
    _sums(torch, B, J, N, C, two, dtype)
