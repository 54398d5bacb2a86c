"""The complex64 panels' sub-blocks of 8 columns (csrc/lu.cu) where they can go
wrong: orders around sub-block and panel edges, pivots scattered over all CTAs
or in one run, rows exchanged at every step, zero columns inside a sub-block.

Bar: the mixed solve refines in FP64, so on these well-conditioned systems the
solution is within 1e-10 of the one the right-hand side was made from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def system(kind, n, rng):
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    if kind == "diag":        # the pivots are the diagonal: one run in one CTA
        A = 0.2 * A + 4 * np.eye(n)
    elif kind == "reversed":  # the pivots come from the other end
        A = 0.2 * A + 4 * np.eye(n)[::-1]
    elif kind == "scattered":
        A = 0.2 * A + 4 * np.eye(n)[rng.permutation(n)]
    elif kind == "ties":      # equal candidates: the lowest row is taken
        A = 0.2 * A / np.abs(A).max() + 4 * np.eye(n)[rng.permutation(n)]
        A[:, ::3] = np.where(np.abs(A[:, ::3]) > 1, A[:, ::3], 0)
    return A


@pytest.mark.parametrize("n", [7, 8, 9, 57, 64, 65, 72, 127, 321, 1025])
@pytest.mark.parametrize("kind", ["diag", "reversed", "scattered", "ties"])
def test_panels(ctx, kind, n):
    rng = np.random.default_rng(n)
    A = system(kind, n, rng)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    y = ctx.solve(A, A @ x, "mixed")
    assert np.linalg.norm(y - x) <= 1e-10 * np.linalg.norm(x)


@pytest.mark.parametrize("n", [7000, 8000])
@pytest.mark.parametrize("kind", ["reversed", "scattered"])
def test_tournament(ctx, kind, n):
    """Tall panels: the tournament's rounds pick from these."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) * (0.2 / n ** 0.5)
    p = torch.arange(n - 1, -1, -1, device="cuda") if kind == "reversed" else \
        torch.randperm(n, device="cuda", generator=g)
    A[torch.arange(n, device="cuda"), p] += 4
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    y = torch.zeros_like(x)
    ctx.solve(A.t().contiguous().t(), b, "mixed", out=y)
    assert (y - x).norm().item() <= 1e-10 * x.norm().item()


@pytest.mark.parametrize("col", [0, 5, 8, 63, 70])
def test_zero_column(ctx, col):
    """A zero column reports the pivot that LAPACK reports."""
    from bem2d_gb300.capi import LapackError
    rng = np.random.default_rng(col)
    A = system("scattered", 200, rng)
    A[:, col] = 0
    with pytest.raises(LapackError) as e:
        ctx.solve(A, np.ones(200, complex), "mixed")
    assert e.value.code == col + 1
