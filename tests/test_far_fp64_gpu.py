"""FP64 far field and potentials (csrc/far_fp64.cu, hankel_tab.cuh) against the
CPU oracle at the edges of their tiles, groups and table octaves.

Tolerance: 1e-12 relative Frobenius (the assembly's bar), plus the conditioning
of e^{i k d}: 4 ulp of the largest argument."""
import numpy as np
import pytest

from bem2d_gb300 import geometry as G
from golden.cases import TRIANGLE

pytestmark = pytest.mark.gpu

QUAD = (3, 5, 0.15)


def tol(k, diam):
    return 1e-12 + 4 * np.finfo(float).eps * abs(k) * diam


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


class Tables(dict):
    def arrays(self):
        return self


def geom(n, bases):
    """Triangle of n elements (n a multiple of 3) with an unknown list: a degree,
    'lin', 'poly4' (runs of 5: groups of 3 and 2), 'basis_major' (groups of 1),
    'mixed' (runs of 1, 2 and 3)."""
    g = G.polygon_uniform(TRIANGLE, n // 3)
    if isinstance(bases, int):
        return Tables(g.add_poly_basis(bases).arrays())
    if bases == "lin":
        return Tables(g.add_lin_basis().arrays())
    if bases == "poly4":
        return Tables(g.add_poly_basis(4).arrays())
    a = Tables(g.add_poly_basis(2).arrays())
    if bases == "basis_major":
        order = np.argsort(a["unk_param"], kind="stable")
    else:
        order = np.array([u for u in range(len(a["unk_elem"]))
                          if a["unk_param"][u] <= a["unk_elem"][u] % 3])
    for key in ("unk_elem", "unk_kind", "unk_param"):
        a[key] = np.ascontiguousarray(a[key][order])
    return a


@pytest.mark.parametrize("n,bases,kernel", [
    (3, 0, "combined"), (33, 0, "combined"), (66, 0, "single"), (99, 0, "double"),
    (39, "lin", "conjdouble"), (66, 2, "combined"), (33, 2, "single"), (24, "poly4", "double"),
    (24, "basis_major", "combined"), (45, "mixed", "conjdouble"), (300, 0, "conjdouble")])
@pytest.mark.parametrize("k", [0.05, 9.0, 40.0 - 6.0j, 11.0 + 2.0j])
def test_matrix_against_oracle(ctx, n, bases, kernel, k):
    from oracle import oracle as O
    a = geom(n, bases)
    A = ctx.discrete_kernel(a, kernel, k, 3.0, QUAD, alpha=1.5, beta=0.5)
    R = O.discrete_kernel(a, kernel, k, 3.0, QUAD, alpha=1.5, beta=0.5)
    assert rel(A, R) < tol(k, 1.0)


@pytest.mark.parametrize("ng", [1, 2, 7, 16])
@pytest.mark.parametrize("bases", [0, 2])
def test_gauss_orders(ctx, ng, bases):
    from oracle import oracle as O
    a = geom(36, bases)
    q = (3, ng, 0.15)
    assert rel(ctx.discrete_kernel(a, "combined", 20.0, 20.0, q),
               O.discrete_kernel(a, "combined", 20.0, 20.0, q)) < tol(20.0, 1.0)


@pytest.mark.parametrize("k", [3000.0, 3000.0 - 0.01j])
def test_arguments_beyond_the_octaves(ctx, k):
    """k d up to 6000 on the unit disk: the last octave and the direct evaluator."""
    from oracle import oracle as O
    a = G.curve_equispaced(G.CIRCLE, 96).add_poly_basis(0)
    assert rel(ctx.discrete_kernel(a, "combined", k, 1.0, QUAD),
               O.discrete_kernel(a, "combined", k, 1.0, QUAD)) < tol(k, 2.0)


@pytest.mark.parametrize("npts", [1, 127, 129, 1000])
@pytest.mark.parametrize("kernel,k", [("single", 30.0), ("combined", 8.0 - 0.5j),
                                      ("double", 0.3), ("conjdouble", 30.0)])
def test_potential_against_oracle(ctx, npts, kernel, k):
    from oracle import oracle as O
    rng = np.random.default_rng(5)
    a = G.kite(77).add_poly_basis(0)
    c = rng.standard_normal(77) + 1j * rng.standard_normal(77)
    p = rng.uniform(2.0, 5.0, (npts, 2))
    u = ctx.potential(a, c, p, kernel, k, 2.0, QUAD)
    v = O.potential(a, c, p, kernel, k, 2.0)
    # a sum of 385 terms of both signs: rounding relative to the terms' size
    size = np.abs(O.potential(a, np.abs(c), p, kernel, k, 2.0)).max() + np.abs(v).max()
    assert np.abs(u - v).max() < 10 * tol(k, 9.0) * size


def test_potential_many_points_equals_few(ctx):
    """Enough points for a single node slice, against the sliced sums."""
    a = G.kite(20).add_poly_basis(0)
    rng = np.random.default_rng(6)
    c = rng.standard_normal(20) + 1j * rng.standard_normal(20)
    p = rng.uniform(2.0, 5.0, (24 * 152 * 128 + 3, 2))
    u = ctx.potential(a, c, p, "single", 5.0, 0.0, QUAD)
    v = ctx.potential(a, c, p[-500:], "single", 5.0, 0.0, QUAD)
    assert np.abs(u[-500:] - v).max() < 1e-13 * np.abs(v).max()
