"""Swaps, U12 and packing between two complex64 panels in one launch
(csrc/lu_tc.cu, tc_step_kernel), and the permutation of all pivots.

Orders where a last panel, a last tile or a short update falls on an edge; row
orders whose swaps chain through the same positions (a cyclic shift moves every
displaced row on at each step) or revisit one row outside the panel.  Bar: the
refined solution within 1e-10 of the one the right-hand side was made from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def order(kind, n, rng):
    if kind == "shift1":
        return np.roll(np.arange(n), 1)
    if kind == "shift64":
        return np.roll(np.arange(n), 64)
    if kind == "pairs":  # the panel's rows and one far row take turns
        p = np.arange(n)
        for i in range(0, n - 1, 2):
            p[i], p[n - 1] = p[n - 1], p[i]
        return p
    return rng.permutation(n)


@pytest.mark.parametrize("n", [65, 96, 128, 129, 191, 193, 320, 321, 449, 833, 1100, 4160])
@pytest.mark.parametrize("kind", ["shift1", "shift64", "pairs", "random"])
def test_step(kind, n):
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    ctx = capi.Context(0)
    rng = np.random.default_rng(n)
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) * (0.2 / n ** 0.5)
    A[torch.arange(n, device="cuda"), torch.from_numpy(order(kind, n, rng)).cuda()] += 3
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    y = torch.zeros_like(x)
    ctx.solve(A.t().contiguous().t(), b, "mixed", out=y)
    ctx.close()
    assert (y - x).norm().item() <= 1e-10 * x.norm().item()
