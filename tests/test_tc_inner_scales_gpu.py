"""The scaled f16 split of the complex64 trailing update (csrc/lu_tc.cu) where the
scales belong to the inner index, and factorisations that make such operands.

Bar of one product, per entry: (K + 4) 2^-22 (|A| |B| + |C|)_ij, the FP32
dot-product bound, as without the scales.

Bar of a refined solve: the matrices have condition numbers below 10 but for
powers of two on rows or columns, which Gaussian elimination in FP32 does not
see; a step of refinement then gains at least 3 digits (n eps cond growth <
1e-3), so backward error 1e-14 takes at most 5 steps and leaves 1e-8 at most in
rows whose weight the norms do not see."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("M,N,K", [(64, 128, 32), (65, 257, 33), (700, 300, 64), (3000, 70, 64),
                                   (300, 900, 256)])
@pytest.mark.parametrize("kind", ["spread", "one_heavy", "columns_only"])
def test_update(ctx, kind, M, N, K):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 31 * K)

    def cm(r, c):
        return torch.randn((c, r), dtype=torch.complex64, device="cuda", generator=g).t()
    A, B, C = cm(M, K), cm(K, N), cm(M, N)
    s = torch.zeros(K, device="cuda")
    if kind == "spread":
        s = torch.randint(-40, 41, (K,), device="cuda", generator=g).float()
    else:
        s[K // 3] = -60
    A = A * 2.0 ** s
    if kind == "columns_only":  # a column of A that does not count beside the others
        B = B * 2.0 ** -10
    else:
        B = B * 2.0 ** -s[:, None]
    A, B, C = (X.t().contiguous().t() for X in (A, B, C))
    c128 = torch.complex128
    ref = C.to(c128) - A.to(c128) @ B.to(c128)
    scale = A.abs().double() @ B.abs().double() + C.abs().double()
    ctx.tc_update(C, A, B)
    assert ((C.to(c128) - ref).abs() <= (K + 4) * 2.0 ** -22 * scale).all()


@pytest.mark.parametrize("n", [200, 300, 1500, 4200])
@pytest.mark.parametrize("rows,s", [(1, 40), (3, 20), (3, 40), (3, 60), (70, 40)])
def test_heavy_rows(ctx, rows, s, n):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) * (0.2 / n ** 0.5)
    A[torch.arange(n, device="cuda"), torch.randperm(n, device="cuda", generator=g)] += 3
    A[torch.randperm(n, device="cuda", generator=g)[:rows]] *= 2.0 ** s
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    y = torch.zeros_like(x)
    ctx.solve(A.t().contiguous().t(), b, "mixed", out=y)
    assert ctx.last_info[1] <= 5
    assert (y - x).norm().item() <= 1e-8 * x.norm().item()
