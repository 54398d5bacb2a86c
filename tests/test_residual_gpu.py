"""The refinement's residual and norms (csrc/lu.cu) where their chunks and routes
change: orders around 1024-row blocks and the chunk lengths of 64, 128 and 256
columns; matrices with and without padding between columns.

Bar: the refined solution within 1e-12 of the one the right-hand side was made
from: a wrong residual entry or norm leaves the single-precision error (1e-6),
or stops or prolongs the refinement."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pad", [(1, 0), (3, 5), (100, 0), (257, 1), (1023, 0), (1025, 3),
                                   (4095, 2), (4096, 0), (8191, 0), (8192, 1)])
def test_refined(n, pad):
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    ctx = capi.Context(0)
    g = torch.Generator(device="cuda").manual_seed(n)
    T = torch.randn((n, n + pad), dtype=torch.complex128, device="cuda", generator=g)
    T *= 0.3 / n ** 0.5
    A = T[:, :n].t()  # column-major, leading dimension n + pad
    A.diagonal().add_(3)
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    y = torch.zeros_like(x)
    ctx.solve(A, b, "mixed", out=y)
    ctx.close()
    assert (y - x).norm().item() <= 1e-12 * x.norm().item()
