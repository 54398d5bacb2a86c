"""The complex128 LU's tensor-core trailing update C -= A B (csrc/lu_oz.cu)
through bem2d_debug_oz_update, against numpy long double.

Bar, per entry (S = A B, rm / cm the largest component of row i of A / column j
of B, one slab per 64 of K, S = sum of slab sums S_q): dropped digit pairs below
2^-52 rm cm a slab, two FP64 roundings of S_q and one of C after each slab."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def dev(torch, a, pad):
    """Column-major device copy with leading dimension rows + pad."""
    r, c = a.shape
    t = torch.zeros((c, r + pad), dtype=torch.complex128, device="cuda")
    t[:, :r] = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    return t[:, :r].t()


def draw(rng, r, c, spread):
    a = rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))
    if spread:  # rows and columns of very different size
        a = a * 2.0 ** rng.integers(-spread, spread + 1, (r, 1)) * 2.0 ** rng.integers(
            -spread, spread + 1, (1, c))
    return a


@pytest.mark.parametrize("M,N,K,pad,spread", [
    (1, 1, 1, 0, 0), (64, 16, 16, 0, 0), (65, 17, 17, 3, 0), (63, 15, 64, 1, 0),
    (130, 33, 48, 0, 0), (200, 300, 64, 5, 0), (96, 40, 100, 2, 0), (70, 50, 64, 0, 200),
    (64, 16, 64, 0, 4), (9, 3000, 33, 0, 0), (3000, 5, 64, 0, 0)])
def test_oz_update(ctx, M, N, K, pad, spread):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(M * 7919 + N * 104729 + K)
    A, B = draw(rng, M, K, spread), draw(rng, K, N, spread)
    if spread == 4:  # all-ones mantissas and powers of two: extreme digits
        A[:, ::2] = np.nextafter(1.0, 0) * (1 - 1j)
        B[::3] = -1.0 + np.nextafter(2.0, 0) * 1j
    C = draw(rng, M, N, 0)
    c = dev(torch, C, pad)
    ctx.oz_update(c, dev(torch, A, pad), dev(torch, B, pad))
    L = np.longdouble
    Ar, Ai, Br, Bi = (x.astype(L) for x in (A.real, A.imag, B.real, B.imag))
    cut = [slice(q, min(q + 64, K)) for q in range(0, K, 64)]
    Sr = [Ar[:, q] @ Br[q] - Ai[:, q] @ Bi[q] for q in cut]
    Si = [Ar[:, q] @ Bi[q] + Ai[:, q] @ Br[q] for q in cut]
    got = c.cpu().numpy()
    rm = np.maximum(abs(A.real), abs(A.imag)).max(1)[:, None]
    cm = np.maximum(abs(B.real), abs(B.imag)).max(0)[None, :]
    for S, g, c0 in ((Sr, got.real, C.real), (Si, got.imag, C.imag)):
        err = np.abs(g.astype(L) - (c0.astype(L) - sum(S))).astype(float)
        size = sum(abs(x) for x in S).astype(float)  # every partial C is below |c0| + size
        bound = 2.0 ** -52 * len(S) * (rm * cm + size + abs(c0))
        assert (err <= bound).all(), (err / bound).max()


def test_oz_update_special_values(ctx):
    """Zero rows and columns leave C; a NaN or an infinity spoils its row or column only."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    A, B, C = draw(rng, 80, 20, 0), draw(rng, 20, 40, 0), draw(rng, 80, 40, 0)
    A[3] = 0
    B[:, 5] = 0
    A[7, 2] = np.nan
    B[4, 9] = np.inf
    A[20] *= 2.0 ** -1040  # subnormal entries count as zero
    c = dev(torch, C, 0)
    ctx.oz_update(c, dev(torch, A, 0), dev(torch, B, 0))
    got = c.cpu().numpy()
    bad = np.zeros((80, 40), bool)
    bad[7] = True
    bad[:, 9] = True
    assert not np.isfinite(got[bad].real).any()
    ok = ~bad
    ref = C - A @ np.where(np.isfinite(B), B, 0)
    assert np.isfinite(got[ok]).all()
    assert np.abs(got[ok] - ref[ok]).max() < 1e-13
    assert (got[3][ok[3]] == C[3][ok[3]]).all() and (got[:, 5][ok[:, 5]] == C[:, 5][ok[:, 5]]).all()
