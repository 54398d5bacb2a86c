"""Bidiagonalisation behind the singular values (csrc/bidiag.cu) over its whole
range: several passes over a CTA's columns with a warp each (orders above some
600), the shared-memory copy of w left out (above 6144), and other GPU work on
the same SMs while its CTAs exchange columns.

Bar: n eps sigma_max, a factor above what the backward stable reduction and the
multisection leave, and at least 1e-12 sigma_max as for the smaller orders."""
import threading

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


@pytest.mark.parametrize("n", [455, 456, 457, 609, 700, 1300])
def test_against_lapack(ctx, n):
    A = crandn(np.random.default_rng(n), n, n)
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(ctx.singular_values(A) - ref).max() <= 1e-12 * ref[0]


def test_known_singular_values_without_the_shared_copy(ctx):
    """n = 6145: H_u diag(sigma) H_v with Householder reflections H."""
    torch = pytest.importorskip("torch")
    n = 6145
    g = torch.Generator(device="cuda").manual_seed(n)
    sig = torch.linspace(2.0, 0.01, n, dtype=torch.float64, device="cuda")
    A = torch.diag(sig.to(torch.complex128))
    for left in (True, False):
        u = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
        u = u / u.norm()
        A = A - 2 * (torch.outer(u, u.conj() @ A) if left else torch.outer(A @ u, u.conj()))
    s = ctx.singular_values(A.t().contiguous().t())
    assert np.abs(s - sig.cpu().numpy()).max() <= 2 * n * np.finfo(float).eps


@pytest.mark.parametrize("n", [130, 512, 700])
def test_beside_other_work(ctx, n):
    """Repeated calls agree bit for bit, idle or beside another context's assembly."""
    from bem2d_gb300 import capi
    from bem2d_gb300 import geometry as G
    A = crandn(np.random.default_rng(n), n, n)
    ref = np.linalg.svd(A, compute_uv=False)
    first = ctx.singular_values(A)
    assert np.abs(first - ref).max() <= 1e-12 * ref[0]
    geom = G.curve_equispaced(G.CIRCLE, 400).add_poly_basis(0)
    stop, other = threading.Event(), capi.Context(0)

    def assemble():
        while not stop.is_set():
            other.discrete_kernel(geom, "combined", 30.0, 30.0, (3, 5, 0.15))

    t = threading.Thread(target=assemble)
    t.start()
    try:
        for _ in range(10):
            assert np.array_equal(ctx.singular_values(A), first)
    finally:
        stop.set()
        t.join()
        other.close()
