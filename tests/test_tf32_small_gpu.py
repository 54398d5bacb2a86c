"""Precision "mixed_tf32" rounds the operands of large trailing updates only: small
ones (fewer than 256 rows or columns) keep the full split, so that a system that
has no others is factored as with "mixed"."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 64, 65, 70, 130, 200, 300, 319])
def test_small_systems_as_mixed(ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    assert np.array_equal(ctx.solve(A, b, "mixed_tf32"), ctx.solve(A, b, "mixed"))


def test_ill_conditioned(ctx):
    """Condition number near 1e10: 10-bit operands leave GMRES-IR nothing to go on."""
    rng = np.random.default_rng(70)
    n = 70
    u = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    A = np.outer(u, u.conj()) * 1e8 + np.eye(n)
    b = A @ (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    x = ctx.solve(A, b, "mixed_tf32")
    r = np.linalg.norm(b - A @ x)
    assert r <= 1e-12 * (np.linalg.norm(A) * np.linalg.norm(x) + np.linalg.norm(b))
