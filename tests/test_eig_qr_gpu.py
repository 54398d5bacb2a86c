"""Pipelined QR (csrc/eig_qr.cu) at the edges of its small blocks (16 rows), of
its sweep counts (8 shifts below 48 rows, 16 above) and on matrices that split,
repeat eigenvalues or stall ordinary shifts.

Bar: eigenvalues as sets within 1e-11 ||A|| of LAPACK's (the bar of
bem2d_eigenvalues), of the known ones for normal matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def distance(a, b):
    """Largest distance in the best one-to-one matching."""
    from scipy.optimize import linear_sum_assignment
    D = np.abs(a[:, None] - b[None, :])
    i, j = linear_sum_assignment(D)
    return D[i, j].max()


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 18, 31, 33, 47, 48, 49, 64, 100, 200])
def test_random(ctx, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    assert distance(ctx.eigenvalues(A), np.linalg.eigvals(A)) < 1e-11 * np.linalg.norm(A, 2)


@pytest.mark.parametrize("n", [17, 40, 90])
def test_normal_with_known_spectrum(ctx, n):
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    d = np.where(rng.random(n) < 0.4, 1.0 + 0.5j, rng.standard_normal(n))  # a multiple eigenvalue
    A = Q @ np.diag(d) @ Q.conj().T
    assert distance(ctx.eigenvalues(A), d) < 1e-11 * np.abs(d).max()


def test_cyclic_shift_and_its_blocks(ctx):
    """Roots of unity: the trailing block is nilpotent, so its shifts are all
    zero; and a block diagonal of such matrices (splits at once)."""
    for sizes in ((60,), (20, 1, 35, 17)):
        n = sum(sizes)
        A = np.zeros((n, n), complex)
        d = []
        at = 0
        for m in sizes:
            A[at:at + m, at:at + m] = np.roll(np.eye(m), 1, 0)
            d.append(np.exp(2j * np.pi * np.arange(m) / m))
            at += m
        assert distance(ctx.eigenvalues(A), np.concatenate(d)) < 1e-11


@pytest.mark.parametrize("scale", [1e-160, 1e150])
def test_scaled(ctx, scale):
    rng = np.random.default_rng(5)
    A = (rng.standard_normal((50, 50)) + 1j * rng.standard_normal((50, 50)))
    ref = np.linalg.eigvals(A)
    assert distance(ctx.eigenvalues(A * scale) / scale, ref) < 1e-11 * np.linalg.norm(A, 2)
