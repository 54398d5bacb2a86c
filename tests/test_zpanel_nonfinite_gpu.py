"""Non-finite entries in the complex128 LU (csrc/lu_zpanel.cu): a NaN is never a
pivot, so the column behind an infinite or spoiled pivot has none and the system
is refused, as by the earlier panels; it must not come back as a solution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from bem2d_gb300 import capi
    c = capi.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("call", ["solve", "noalloc"])
@pytest.mark.parametrize("n", [5, 20, 33, 70, 200, 600])
@pytest.mark.parametrize("value", [np.inf, -np.inf, 1j * np.inf, np.nan])
def test_refused(ctx, value, n, call):
    from bem2d_gb300 import capi
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (0.3 / n ** 0.5)
    A += 3 * np.eye(n)[rng.permutation(n)]
    A[1, 2] = value
    b = np.ones(n, complex)
    with pytest.raises(capi.LapackError):
        ctx.solve(A, b, "fp64") if call == "solve" else ctx.solve_noalloc(A, b)
