"""Geometries whose element pairs are all identical or adjacent: nothing is left to
the far field (no launch, no table of a complex wavenumber).  Against the oracle,
1e-12 relative Frobenius, as for the other geometries."""
import numpy as np
import pytest

from bem2d_gb300 import geometry as G

pytestmark = pytest.mark.gpu

Q = (3, 5, 0.15)
GEOMS = {
    "one": lambda: G.line_uniform((0.0, 0.0), (1.0, 0.5), 1),
    "two": lambda: G.line_uniform((0.0, 0.0), (1.0, 0.5), 2),
    "triangle": lambda: G.polygon_uniform([(0.0, 0.0), (1.0, 0.0), (0.3, 0.8)], 1),
}


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("k", [5.0, 4.0 - 1.0j, 4.0 + 2.0j])
@pytest.mark.parametrize("degree", [0, 1, 4])
@pytest.mark.parametrize("name", sorted(GEOMS))
def test_matrix(ctx, name, degree, k):
    from oracle import oracle as O
    g = GEOMS[name]().add_poly_basis(degree)
    for kernel in ("single", "combined"):
        n = len(g.arrays()["unk_elem"])
        out = np.full((n, n), np.nan, complex, order="F")  # every entry is written
        before = ctx.launches
        A = ctx.discrete_kernel(g, kernel, k, 2.0, Q, out=out)
        assert ctx.launches - before <= 3  # node table, near field, scan for NaN
        ref = O.discrete_kernel(g, kernel, k, 2.0, Q)
        assert np.linalg.norm(A - ref) <= 1e-12 * np.linalg.norm(ref)
