"""The scaled f16 split of the complex64 trailing update (csrc/lu_tc.cu) where
its scales matter, through bem2d_debug_tc_update against a complex128 product.

Bar, per entry: (K + 4) 2^-22 (|A| |B| + |C|)_ij, the FP32 dot-product bound:
the split keeps 22 bits of an entry within 2^-16 of its row's (column's) largest
and 2^-40 of that largest otherwise, so rows, columns or whole operands of any
size float can hold must not lose to it, nor random entries over 4 decades."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("M,N,K", [(64, 128, 32), (65, 257, 33), (700, 300, 64), (300, 900, 256)])
@pytest.mark.parametrize("kind", ["rows", "cols", "entries", "tiny", "huge", "zero", "pow2"])
def test_scales(ctx, kind, M, N, K):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 31 * K)

    def cm(r, c):
        return torch.randn((c, r), dtype=torch.complex64, device="cuda", generator=g).t()

    def u(r, c):
        return torch.rand((c, r), device="cuda", generator=g).t()
    A, B, C = cm(M, K), cm(K, N), cm(M, N)
    if kind == "rows":
        A = A * 10 ** (-12 * u(M, 1))
    elif kind == "cols":
        B = B * 10 ** (-12 * u(1, N))
    elif kind == "entries":
        A, B = A * 10 ** (-4 * u(M, K)), B * 10 ** (-4 * u(K, N))
    elif kind == "tiny":
        A, B, C = A * 1e-18, B * 1e-18, C * 1e-36
    elif kind == "huge":
        A, B, C = A * 1e17, B * 1e17, C * 1e34
    elif kind == "zero":
        A[::3] = 0
        B[:, ::5] = 0
    else:  # magnitudes at the edges of the scaling interval
        A = torch.complex(torch.full((K, M), 2.0, device="cuda").t(),
                          torch.full((K, M), 2.0 - 2.0 ** -23, device="cuda").t())
    A, B, C = (X.t().contiguous().t() for X in (A, B, C))
    c128 = torch.complex128
    ref = C.to(c128) - A.to(c128) @ B.to(c128)
    scale = A.abs().double() @ B.abs().double() + C.abs().double()
    ctx.tc_update(C, A, B)
    assert ((C.to(c128) - ref).abs() <= (K + 4) * 2.0 ** -22 * scale).all()
