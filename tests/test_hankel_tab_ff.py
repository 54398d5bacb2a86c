"""The float-float table evaluator of the mixed far field
(csrc/hankel_tab_ff.cuh): accuracy on the host, and the far field on every route
it takes (table intervals in shared or global memory, arguments beyond the
table, other rule sizes)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hktab") / "libhktab.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=on",
                    "-I" + os.path.join(ROOT, "bem2d_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "hankel_tab_ff_host.cpp"), "-o", out],
                   check=True)
    return ctypes.CDLL(out)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _ff_round(x):
    hi = x.astype(np.float32).astype(np.float64)
    return hi + (x - hi).astype(np.float32).astype(np.float64)


def test_table_against_mpmath(lib):
    """H0 and H1/x at 4 <= x < 4096, all octaves and interval edges: relative
    error within 3e-14, the bar of the general evaluator (about eight roundings
    of 2^-48 in E, the polynomial and their product)."""
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 40
    rng = np.random.default_rng(8)
    edges = np.concatenate([2.0 ** e * (1 + np.arange(0, 128, 9) / 128) for e in range(2, 12)])
    x = _ff_round(np.concatenate([2 ** rng.uniform(2, 12, 900), edges, edges * (1 + 2.0 ** -23),
                                  np.nextafter(np.float32(edges[1:]), np.float32(0)).astype(float),
                                  np.array([np.nextafter(np.float32(4096), np.float32(0))], float)]))
    o = np.zeros((len(x), 4))
    assert lib.hankel_tab_ff_host(ctypes.c_int(len(x)), _p(x), _p(o)) == 0
    h0, h1 = o[:, 0] + 1j * o[:, 1], o[:, 2] + 1j * o[:, 3]
    r0 = np.array([complex(mp.hankel1(0, mp.mpf(float(v)))) for v in x])
    r1 = np.array([complex(mp.hankel1(1, mp.mpf(float(v))) / mp.mpf(float(v))) for v in x])
    assert (np.abs(h0 - r0) / np.abs(r0)).max() < 3e-14
    assert (np.abs(h1 - r1) / np.abs(r1)).max() < 3e-14


def test_outside_the_table(lib):
    """What the bin test must leave to the general evaluator."""
    x = np.array([0.0, 1e-30, 3.9999, 4096.0, 1e30, np.inf, -5.0, np.nan])
    o = np.zeros((len(x), 4))
    assert lib.hankel_tab_ff_host(ctypes.c_int(len(x)), _p(x), _p(o)) == len(x)


def test_sqrt(lib):
    """ff_sqrt within 2^-46 (its result is one float-float rounding, 2^-48,
    plus the single-precision rounding of the correction, 2^-47)."""
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 40
    rng = np.random.default_rng(9)
    x = _ff_round(2 ** rng.uniform(-20, 40, 3000))
    o = np.zeros_like(x)
    lib.sqrt_ff_host(ctypes.c_int(len(x)), _p(x), _p(o))
    err = [abs(float(mp.mpf(float(a)) / mp.sqrt(mp.mpf(float(v))) - 1)) for a, v in zip(o, x)]
    assert max(err) < 2.0 ** -46


def _geom(name):
    from bem2d_gb300 import geometry as G
    if name == "fine":      # small steps of k|x - y|: table intervals in shared memory
        return G.kite(700).add_poly_basis(0)
    if name == "coarse":    # a tile's arguments span octaves: intervals from the global table
        return G.kite(70).add_poly_basis(0)
    return G.kite(33).add_poly_basis(2)  # runs of unknowns of one element


@pytest.mark.gpu
@pytest.mark.parametrize("name,k,q", [
    ("fine", 30.0, (3, 5, 0.15)), ("fine", 3000.0, (3, 5, 0.15)), ("coarse", 40.0, (3, 5, 0.15)),
    ("coarse", 0.05, (3, 5, 0.15)), ("poly", 9.0, (3, 3, 0.15)), ("poly", 900.0, (2, 8, 0.15)),
    ("coarse", 25.0, (0, 64, 0.15))])
@pytest.mark.parametrize("kernel", ["single", "double", "conjdouble", "combined"])
def test_far_field_routes(kernel, name, k, q):
    """Mixed assembly against the FP64 one (relative Frobenius): 1e-13 per
    evaluation plus the phase's share, x 2^-46 at the largest argument (the
    float-float x carries about five roundings of 2^-48); the normal product of
    the double layers cancels against |x - y|: a factor 4 on both."""
    from bem2d_gb300 import capi
    g = _geom(name)
    ctx = capi.Context(0)
    A = ctx.discrete_kernel(g, kernel, k, k, q, alpha=1.0, beta=0.0)
    M, M32 = ctx.discrete_kernel_mixed(g, kernel, k, k, q, alpha=1.0, beta=0.0)
    ctx.close()
    bound = 4 * (1e-13 + 3.6 * k * 2.0 ** -46)  # the kite's diameter is below 3.6
    assert np.linalg.norm(M - A) <= bound * np.linalg.norm(A)
    assert np.linalg.norm(M32.astype(np.complex128) - M) <= 1e-7 * np.linalg.norm(M)
