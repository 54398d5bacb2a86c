"""Digit products (csrc/oz.cuh) of operands at the ends of the range of a double:
entries below 2^-1022 keep their bits, as in the FP64 arithmetic before.

Bar of a product: the terms' rounding, 2 K + 4 units of 2^-53 of |A| |B| + |C|, and
of the smallest subnormal, 2^-1074, each.  Bar of a solve: as for the same matrix
without its factor (condition number below 10, n = 200): 1e-12."""
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


@pytest.mark.parametrize("s", [-1050, -1030, -1020, -1000, 990])
@pytest.mark.parametrize("M,N,K", [(64, 16, 64), (70, 33, 20)])
def test_update(ctx, M, N, K, s):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(M + 2000 - s)
    A, B, C = crandn(rng, M, K), crandn(rng, K, N), crandn(rng, M, N)
    # scaled in two steps: 2^s alone may be subnormal
    h = s // 2
    B, C = B * 2.0 ** h * 2.0 ** (s - h), C * 2.0 ** h * 2.0 ** (s - h)
    dev = [torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t() for x in (C, A, B)]
    ctx.oz_update(*dev)
    L = np.longdouble
    up = L(2.0) ** -s
    got, Bs, Cs = dev[0].cpu().numpy(), B, C
    size = np.abs(A) @ np.full((K, N), 5.0) + 5  # |B| and |C| are below 5 2^s
    bound = (2 * K + 4) * (2.0 ** -53 * size + 2.0 ** min(-1074.0 - s, 0.0) * (s < -900))
    Ar, Ai = A.real.astype(L), A.imag.astype(L)
    Br, Bi = Bs.real.astype(L) * up, Bs.imag.astype(L) * up
    for g, c, S in ((got.real, Cs.real, Ar @ Br - Ai @ Bi), (got.imag, Cs.imag, Ar @ Bi + Ai @ Br)):
        err = np.abs(g.astype(L) * up - (c.astype(L) * up - S)).astype(float)
        assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("s", [-1005, -1000, -960, -500, 500, 1000])
def test_solve(ctx, s):
    rng = np.random.default_rng(7)
    n = 200
    A = crandn(rng, n, n) * (0.2 / n ** 0.5) + 3 * np.eye(n)[rng.permutation(n)]
    x = crandn(rng, n)
    y = ctx.solve(A * 2.0 ** s, (A @ x) * 2.0 ** s, "fp64")
    assert np.abs(y - x).max() <= 1e-12 * np.abs(x).max()
