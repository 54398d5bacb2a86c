"""Calls whose tensor-core operands do not fit beside what the device already
holds: another allocation leaves a few hundred MB, in steps, so that some steps fall
between what a call cannot do without and what it would like.

Bars as for the same calls with room: n eps for the backward error of a Gaussian
system (its growth is far below n), 1e-11 of the Hermitian part's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Leave:
    """All but `size` bytes of the device's memory taken, for a while."""

    def __init__(self, torch, size):
        self.torch, self.size = torch, size

    def __enter__(self):
        self.torch.cuda.empty_cache()
        free = self.torch.cuda.mem_get_info()[0]
        self.hold = self.torch.empty(free - self.size, dtype=self.torch.uint8, device="cuda")

    def __exit__(self, *_):
        del self.hold
        self.torch.cuda.empty_cache()


def with_all_kernels_loaded(torch, capi, B=None, th=None):
    """Kernels are loaded by their first launch, which takes device memory."""
    ctx = capi.Context(0)
    rng = np.random.default_rng(1)
    A = rng.standard_normal((200, 200)) + 1j * rng.standard_normal((200, 200))
    ctx.solve(A, np.ones(200, complex), "fp64")
    ctx.solve_noalloc(A, np.ones(200, complex))  # the updates without operands
    for precision in ("fp64", "mixed"):
        ctx.num_range_lmax(A, np.array([0.3]), precision=precision)
        if B is not None:
            ctx.num_range_lmax(B, th, precision=precision)
    ctx.close()


def test_fp64_solve():
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    n = 4096  # the factor: 256 MB; its diagonal blocks' inverses 8, packed operands 18
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g).t()
    b = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    norms = float(torch.linalg.norm(A)), float(torch.linalg.norm(b))
    with_all_kernels_loaded(torch, capi)
    done = []
    for left in range(264, 340, 4):
        x = torch.zeros_like(b)
        ctx = capi.Context(0)
        try:
            with Leave(torch, left * MB):
                ctx.solve(A, b, "fp64", out=x)
        except capi.Bem2dError as e:
            assert "out of memory" in str(e), e
            assert not done  # what fitted before fits with more
            continue
        finally:
            ctx.close()
        done.append(left)
        r = float(torch.linalg.norm(b - A @ x))
        assert r <= n * np.finfo(float).eps * (norms[0] * float(torch.linalg.norm(x)) + norms[1])
    assert done and done[0] < 256 + 8 + 18  # less than all of them


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_num_range(precision):
    torch = pytest.importorskip("torch")
    from bem2d_gb300 import capi
    n, th = 1500, np.array([0.1, 1.2, 2.9])
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda().t()
    ref = []
    for t in th:
        z = np.exp(1j * t)
        w = np.linalg.eigvalsh(0.5 * (z * A + np.conj(z) * A.conj().T))
        ref.append((w[-1], np.abs(w).max()))
    with_all_kernels_loaded(torch, capi, dA, th)
    launches = set()
    for left in list(range(40, 280, 16)) + [600]:
        ctx = capi.Context(0)
        try:
            with Leave(torch, left * MB):
                got = ctx.num_range_lmax(dA, th, tol=1e-12, precision=precision)
        except capi.Bem2dError as e:
            assert "out of memory" in str(e), e
            continue
        finally:
            launches.add(ctx.launches)
            ctx.close()
        for v, (w, size) in zip(got, ref):
            assert abs(v - w) <= 1e-11 * size
    assert len(launches - {0}) >= 3  # whole, and two sizes of row blocks
