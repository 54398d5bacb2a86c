"""The complex64 triangular solve (csrc/lu.cu, trisolve64_kernel) repeated beside
other GPU work: its messages between CTAs must not depend on how long they take.

Orders whose last round of blocks leaves CTAs without a block after the others'
(one block short of, at and past a multiple of the 16 CTAs).  Refined solutions
of repeated calls agree bit for bit: every step is in a fixed order."""
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 100, 960, 1000, 1024, 1025, 1088, 2000])
def test_repeats_beside_other_work(n):
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    from bem2d_gb300 import geometry as G
    ctx, other = capi.Context(0), capi.Context(0)
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) * (0.3 / n ** 0.5)
    A[torch.arange(n, device="cuda"), torch.randperm(n, device="cuda", generator=g)] += 3
    x = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    b = A @ x
    Ac = A.t().contiguous().t()
    first, y = torch.zeros_like(x), torch.zeros_like(x)
    ctx.solve(Ac, b, "mixed", out=first)
    assert (first - x).norm().item() <= 1e-10 * x.norm().item()
    geom = G.curve_equispaced(G.CIRCLE, 400).add_poly_basis(0)
    stop = threading.Event()

    def assemble():
        while not stop.is_set():
            other.discrete_kernel(geom, "combined", 30.0, 30.0, (3, 5, 0.15))

    t = threading.Thread(target=assemble)
    t.start()
    try:
        for _ in range(40):
            ctx.solve(Ac, b, "mixed", out=y)
            assert torch.equal(y, first)
    finally:
        stop.set()
        t.join()
        other.close()
        ctx.close()
