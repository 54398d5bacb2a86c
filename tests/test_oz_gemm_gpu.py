"""Numerical range through the digit products (csrc/oz_gemm.cu) at the edges of
their tiles (64 rows, 32 columns), K steps (16) and accumulator chunks (128), and
with rows and columns of very different size, zeros and non-finite entries.

Bar: each lambda_max within 1e-11 of the Hermitian part's 2-norm (LAPACK zheev),
the scan's own stopping bound at tol 1e-12 with a margin of ten."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def lmax(A, th):
    z = np.exp(1j * th)
    H = 0.5 * (z * A + np.conj(z) * A.conj().T)
    w = np.linalg.eigvalsh(H)
    return w[-1], np.abs(w).max()


@pytest.mark.parametrize("n,nang,spread", [
    (1, 1, 0), (5, 3, 0), (15, 33, 0), (16, 32, 0), (17, 31, 0), (64, 1, 0), (65, 40, 0),
    (127, 5, 0), (129, 65, 0), (257, 7, 0), (300, 96, 0), (100, 20, 25)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_num_range(ctx, n, nang, spread, precision):
    rng = np.random.default_rng(n + nang)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if spread:
        A = A * 2.0 ** -rng.integers(0, spread, (n, 1)) * 2.0 ** -rng.integers(0, spread, (1, n))
    th = 2 * np.pi * np.arange(nang) / nang + 0.1
    got = ctx.num_range_lmax(A, th, tol=1e-12, precision=precision)
    for g, t in zip(got, th):
        ref, size = lmax(A, t)
        assert abs(g - ref) <= 1e-11 * size


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_rows(ctx, precision):
    rng = np.random.default_rng(2)
    A = rng.standard_normal((40, 40)) + 1j * rng.standard_normal((40, 40))
    A[3] = 0
    A[:, 7] = 0
    th = np.array([0.0, 1.0, 2.0])
    got = ctx.num_range_lmax(A, th, tol=1e-12, precision=precision)
    for g, t in zip(got, th):
        ref, size = lmax(A, t)
        assert abs(g - ref) <= 1e-11 * size
