"""Singular values (csrc/bidiag.cu) of matrices whose squares leave the range of a
double, as a whole or in a remainder of the reduction.

Bar: 1e-12 sigma_max as for ordinary matrices; scaling by powers of two commutes
with every rounding of the reduction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def crandn(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("n", [1, 2, 50, 300])
@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -560, 2.0 ** -200, 2.0 ** 200, 2.0 ** 560,
                                   2.0 ** 1000])
def test_scaled(ctx, scale, n):
    A = crandn(np.random.default_rng(n), n, n)
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(ctx.singular_values(A * scale) / scale - ref).max() <= 1e-12 * ref[0]


@pytest.mark.parametrize("tiny", [0.0, 1e-170j, (1 + 1j) * 1e-200, 1e-310j])
def test_tiny_remainders(ctx, tiny):
    """Blocks that no other entry reaches, below and beside ordinary ones."""
    rng = np.random.default_rng(2)
    for n in (2, 3, 40):
        A = np.zeros((n, n), complex)
        m = n // 2
        A[:m, :m] = crandn(rng, m, m)
        A[m:, m:] = tiny * (1 + rng.random((n - m, n - m)))
        ref = np.linalg.svd(A, compute_uv=False)
        assert np.abs(ctx.singular_values(A) - ref).max() <= 1e-12 * ref[0]


def test_zero_matrix(ctx):
    assert (ctx.singular_values(np.zeros((20, 20), complex)) == 0).all()
