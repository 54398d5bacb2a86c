"""The complex64 triangular solve in one cluster (csrc/lu.cu, trisolve64_kernel)
at the orders where its blocks, CTAs and rounds change: fewer blocks than CTAs,
one, two and more blocks per CTA, ragged last blocks, up to the last order
before the wavefront solve.

Bar: the refined solution within 1e-10 of the one the right-hand side was made
from, in few enough steps that the mixed path does not give up (the systems are
well conditioned)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 129, 511, 575, 577, 1023, 1024, 1025, 1089,
                               2048, 2049, 3137, 5000, 8191])
def test_solve(n):
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    ctx = capi.Context(0)
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) * (0.3 / n ** 0.5)
    A[torch.arange(n, device="cuda"), torch.randperm(n, device="cuda", generator=g)] += 3
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    y = torch.zeros_like(x)
    for _ in range(3):
        ctx.solve(A.t().contiguous().t(), b, "mixed", out=y)
        assert (y - x).norm().item() <= 1e-10 * x.norm().item()
    ctx.close()
