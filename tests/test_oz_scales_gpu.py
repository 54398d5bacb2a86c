"""The complex128 LU's tensor-core update (csrc/lu_oz.cu) where rows, columns,
inner indices or single entries lie many powers of two apart.

Bar of one product, per entry with T the largest of |a_ik| |b_kj| (components)
over a slab of 64: where the digits serve, T is at least 2^-10 in exponents, so
at least 2^-12 in value, of row's largest x column's largest, and the dropped
digit pairs are below 2^-52 of that: 2^-40 T; else the FP64 sum.  Beside it
2 K + 4 roundings of |A| |B| + |C|.

Bar of a solve: scaling rows and columns by powers of two commutes with every
rounding of Gaussian elimination but for the choice of pivots; the matrices have
condition numbers below 10, growth of n / 10 and n eps cond growth < 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


def crandn(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def pow2(rng, span, *shape):
    return 2.0 ** rng.integers(-span, span + 1, shape)


@pytest.mark.parametrize("M,N,K", [(3, 2, 2), (64, 16, 64), (65, 17, 33), (200, 130, 64),
                                   (130, 50, 100)])
@pytest.mark.parametrize("kind", ["inner", "entries", "sparse", "two", "decay"])
def test_update(ctx, kind, M, N, K):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(M + 31 * N + 977 * K)
    A, B, C = crandn(rng, M, K), crandn(rng, K, N), crandn(rng, M, N)
    if kind == "inner":  # a scale that belongs to k, undone in B
        s = pow2(rng, 200, K)
        A, B = A * s, B / s[:, None]
    elif kind == "entries":
        A, B, C = A * pow2(rng, 40, M, K), B * pow2(rng, 40, K, N), C * 2.0 ** -70
    elif kind == "sparse":  # mostly zeros, large and small entries that never meet
        A, B = A * (rng.random((M, K)) < 0.1), B * (rng.random((K, N)) < 0.1)
        A[:, ::2] *= 2.0 ** 50
        B[::2] *= 2.0 ** -90
        C *= 2.0 ** -60
    elif kind == "two":  # a_i = (1, tiny), b_j = (tiny, 1)
        A[:, 1:] *= 2.0 ** -60
        B[0] *= 2.0 ** -60
        C *= 2.0 ** -60
    else:  # exponentially decaying couplings
        i, k, j = (np.arange(x)[:, None] for x in (M, K, N))
        A, B = A * 2.0 ** -(i + k.T), B * 2.0 ** -(k + j.T)
        C *= 2.0 ** -(i + j.T)
    dev = [torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t() for x in (C, A, B)]
    ctx.oz_update(*dev)
    L = np.longdouble
    Ar, Ai, Br, Bi = (x.astype(L) for x in (A.real, A.imag, B.real, B.imag))
    got = dev[0].cpu().numpy()
    ca, cb = (np.maximum(abs(x.real), abs(x.imag)) for x in (A, B))
    size = (ca @ cb) * 2 + abs(C)
    top = sum((ca[:, q:q + 64, None] * cb[None, q:q + 64]).max(1) for q in range(0, K, 64))
    bound = 2.0 ** -40 * top + (2 * K + 4) * EPS * size
    for g, c, S in ((got.real, C.real, Ar @ Br - Ai @ Bi), (got.imag, C.imag, Ar @ Bi + Ai @ Br)):
        err = np.abs(g.astype(L) - (c.astype(L) - S)).astype(float)
        assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("n", [130, 300, 700])
@pytest.mark.parametrize("kind", ["rows", "cols", "both", "heavy_col", "heavy_row"])
def test_solve(ctx, kind, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    A = crandn(rng, n, n) * (0.2 / n ** 0.5) + 3 * np.eye(n)[rng.permutation(n)]
    x = crandn(rng, n)
    r, c = np.ones(n), np.ones(n)
    if kind in ("rows", "both"):
        r = pow2(rng, 40, n)
    if kind in ("cols", "both"):
        c = pow2(rng, 40, n)
    if kind == "heavy_col":
        c[[5, n // 2, n - 3]] = 2.0 ** 60
    if kind == "heavy_row":
        r[[5, n // 2, n - 3]] = 2.0 ** 60
    b = (A @ x) * r
    y = ctx.solve(A * r[:, None] * c, b, "fp64") * c
    assert np.abs(y - x).max() <= 1e-10 * np.abs(x).max()
