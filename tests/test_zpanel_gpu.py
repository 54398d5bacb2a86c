"""Complex128 LU panels (csrc/lu_zpanel.cu) at the edges of their blocks (16
columns), warps (32 rows), clusters (16 x 256 rows, one row per thread; two up
to 8192) and of the taller panels' fallback, through bem2d_solve_system.

Bar: LU with partial pivoting is backward stable; the normwise backward error of
Gaussian systems stays below n eps (their growth factor is far below n)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 48, 64, 79, 81, 127, 130, 513, 1030, 4096,
                               4100, 8193, 8300])
def test_backward_error(ctx, n):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g).t()
    b = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    x = torch.zeros_like(b)
    ctx.solve(A, b, "fp64", out=x)
    r = torch.linalg.norm(b - A @ x)
    berr = float(r / (torch.linalg.norm(A) * torch.linalg.norm(x) + torch.linalg.norm(b)))
    assert berr <= max(n, 8) * np.finfo(float).eps


def test_pivoting_is_needed_and_ties_go_to_the_first_row(ctx):
    """Zero diagonal, equal magnitudes, rows of very different size: as LAPACK."""
    rng = np.random.default_rng(3)
    for n in (20, 70):
        A = rng.integers(-1, 2, (n, n)) + 1j * rng.integers(-1, 2, (n, n))
        A = A + 0.5 * np.eye(n)[::-1] + 0.25 * np.roll(np.eye(n), 1, 0)
        A *= 2.0 ** rng.integers(-200, 200, (n, 1))
        b = A @ np.ones(n)
        x = ctx.solve(A, b, "fp64")
        assert np.abs(x - np.linalg.solve(A, b)).max() < 1e-9


@pytest.mark.parametrize("n,col", [(20, 0), (20, 17), (70, 33), (200, 150)])
def test_zero_pivot_is_reported_at_its_column(ctx, n, col):
    from bem2d_gb300 import capi
    rng = np.random.default_rng(4)
    A = np.triu(rng.standard_normal((n, n)) + 2 * np.eye(n)).astype(complex)
    A[col, col] = 0.0
    with pytest.raises(capi.LapackError) as e:
        ctx.solve(A, np.ones(n, complex), "fp64")
    assert e.value.code == col + 1
