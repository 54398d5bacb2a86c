"""Timed cases of the framework: the calls that scattering, norm, numerical-range
and resonance programs make, through bem2d_gb300.capi.

Each case is a dict of plain values.  `kind` names the program:

  scatter    Discretize() + Solve() of one sound-soft problem
  sweep      many wavenumbers of one obstacle in one batched call
  solve      SolveSystem on a system matrix that is already on the device
  assemble   DiscreteKernel alone, with polynomial bases
  normcond   assembly, mass matrix, ChangeBasis, ||A|| and cond(A)
  numrange   assembly, mass matrix, ChangeBasis, numerical range
  field      the potential of a density on a grid of points
  resonance  one point of a complex-k scan: assembly and singular values
  spectrum   assembly, mass matrix, ChangeBasis, eigenvalues

Wavenumbers (within 1 %), incident directions and right-hand sides come from
the seed; sizes come from the case.  One Context serves every state, as a
program keeps one for all its problems; matrices stay on the device.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bem2d_gb300 import capi
from bem2d_gb300 import geometry as G

QUAD = (3, 5, 0.15)  # the library's default QuadOption {L, N, sigma}
NR_TOL = 1e-11

SQUARE = [(0.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.0, 1.0)]
LSHAPE = [(0.0, 0.0), (1.0, 0.0), (1.0, 0.5), (0.5, 0.5), (0.5, 1.0), (0.0, 1.0)]
TRIANGLE = [(0.0, 0.0), (1.0, 0.0), (0.3, 0.8)]
# trapping domain of the resonance scan
TRAP = [(0.0, 0.0), (-1.0, 0.0), (-1.0, -0.69), (0.69, -0.69), (0.69, 1.31), (-1.0, 1.31),
        (-1.0, 0.62), (0.0, 0.62)]
POLYGONS = {"square": SQUARE, "lshape": LSHAPE, "triangle": TRIANGLE, "trap": TRAP}
CURVES = {"disk": (G.CIRCLE, (0.0, 0.0, 0.0, 0.0)), "kite": (G.KITE, (0.0, 0.0, 0.0, 0.0)),
          "ellipse": (G.ELLIPSEARC, (2.0, 1.0, 0.0, 2 * G.PI))}
PERIMETER = {"disk": 2 * math.pi, "kite": 9.324, "ellipse": G.ELLIPSE21_PERIMETER, "square": 4.0,
             "lshape": 4.0, "triangle": 2.917, "trap": 10.0}


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # the smallest program: unit disk, the library's FP64 default
        dict(name="disk160_fp64", kind="scatter", shape="disk", n=160, graded=0, k=10.0,
             precision="fp64"),
        # one ordinary solve, in the library's default precision and in the mixed one
        dict(name="kite2048_fp64", kind="scatter", shape="kite", n=2048, graded=0, k=100.0,
             precision="fp64"),
        dict(name="kite2048_mixed", kind="scatter", shape="kite", n=2048, graded=0, k=100.0,
             precision="mixed"),
        # the largest single solve: graded corners, high wavenumber
        dict(name="lshape16384_mixed", kind="scatter", shape="lshape", n=16384, graded=8, k=500.0,
             precision="mixed"),
        # a wavenumber sweep, N_k = 309 ... 3084 (uneven)
        dict(name="sweep256_mixed", kind="sweep", nk=256, k_lo=20.0, k_hi=200.0,
             precision="mixed"),
        # SolveSystem with a matrix the program holds (odd order)
        dict(name="solve3001_fp64", kind="solve", shape="kite", n=3001, k=140.0,
             precision="fp64"),
        # DiscreteKernel with PolBasis(2), as the numerical-range programs assemble (odd order)
        dict(name="poly2_2403_fp64", kind="assemble", shape="triangle", n=801, degree=2, k=100.0,
             kernel="conjdouble"),
        # the norm / condition number study, graded square
        dict(name="normcond8192_mixed", kind="normcond", shape="square", n=8192, graded=8,
             k=200.0, precision="mixed"),
        # the numerical-range study
        dict(name="numrange2048_mixed", kind="numrange", shape="square", n=2048, graded=0, k=50.0,
             nang=360, precision="mixed"),
        # EvalSol on the plotting grid
        dict(name="field200x200", kind="field", shape="kite", n=1024, k=50.0, grid=200),
        # one wavenumber of the resonance scan
        dict(name="trap512_resonance", kind="resonance", shape="trap", n=512, k=6.0, kim=-1.0),
        # the spectrum of the combined operator
        dict(name="triangle255_spectrum", kind="spectrum", shape="triangle", n=255, k=10.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scatter", "scatter", "scatter", "sweep", "solve", "assemble", "normcond",
                       "numrange", "field", "resonance", "spectrum"])
    if kind == "sweep":
        lo = rng.uniform(15.0, 60.0)
        return dict(kind=kind, nk=_log(rng, 8, 96), k_lo=round(lo, 3),
                    k_hi=round(lo * rng.uniform(1.2, 3.3), 3),
                    precision=rng.choice(["mixed", "mixed", "mixed_tf32"]))
    if kind == "resonance":
        return dict(kind=kind, shape="trap", n=_log(rng, 96, 600), k=round(rng.uniform(2.0, 12.0), 3),
                    kim=round(-rng.uniform(0.05, 2.0), 3))
    if kind == "spectrum":
        return dict(kind=kind, shape="triangle", n=_log(rng, 48, 300), k=round(rng.uniform(2.0, 15.0), 3))
    if kind == "numrange":
        prec = rng.choice(["mixed", "mixed", "fp64"])
        n = _log(rng, 128, 2048 if prec == "mixed" else 900)
        return dict(kind=kind, shape="square", n=n, graded=0, k=round(n / 40.0, 3),
                    nang=_log(rng, 24, 360), precision=prec)
    if kind == "normcond":
        prec = rng.choice(["mixed", "mixed", "fp64"])
        n = _log(rng, 256, 8192 if prec == "mixed" else 2500)
        return dict(kind=kind, shape=rng.choice(["square", "lshape"]), n=n,
                    graded=rng.choice([0, 3, 8]), k=round(n / 40.0, 3), precision=prec)
    shape = rng.choice(["disk", "kite", "ellipse", "square", "lshape"])
    ppw = rng.uniform(8.0, 16.0)
    if kind == "field":
        n = _log(rng, 128, 1500)
        shape = rng.choice(["disk", "kite", "ellipse"])
        return dict(kind=kind, shape=shape, n=n,
                    k=round(2 * math.pi * n / (ppw * PERIMETER[shape]), 3),
                    grid=_log(rng, 30, 200))
    if kind == "assemble":
        n, degree = _log(rng, 64, 3000), rng.choice([0, 1, 2])
        n = max(24, n // (degree + 1))
        return dict(kind=kind, shape=shape, n=n, degree=degree,
                    k=round(2 * math.pi * n / (ppw * PERIMETER[shape]), 3),
                    kernel=rng.choice(["single", "double", "conjdouble", "combined"]))
    prec = rng.choice(["fp64", "mixed", "mixed", "mixed_tf32"])
    n = _log(rng, 100, 3200 if prec == "fp64" else 9000)
    k = round(2 * math.pi * n / (ppw * PERIMETER[shape]), 3)
    if kind == "solve":
        return dict(kind=kind, shape=shape, n=n, k=k, precision=prec)
    return dict(kind=kind, shape=shape, n=n,
                graded=rng.choice([0, 3, 8]) if shape in POLYGONS else 0, k=k, precision=prec)


# ---- geometry tables -----------------------------------------------------------
def _curve_tables(shape, n):
    """n elements equispaced in the parameter of a closed curve, one constant
    basis function each, as the flat tables the library takes."""
    kind, cp = CURVES[shape]
    i = np.arange(n)
    param = np.zeros((n, 8))
    param[:, 0], param[:, 1], param[:, 2:6] = i / n, (i + 1) / n, cp
    return dict(kind=np.full(n, kind, np.int32), param=param, index=i.astype(np.int64),
                next=((i + 1) % n).astype(np.int64), prev=((i - 1) % n).astype(np.int64),
                unk_elem=i.astype(np.int32), unk_kind=np.zeros(n, np.int32),
                unk_param=np.zeros(n))


def _tables(shape, n, graded=0, degree=0):
    """Element tables of about n elements (exactly n on curves, and on
    polygons too: the coarse cells are dealt out to the sides)."""
    if shape in CURVES:
        t = _curve_tables(shape, n)
    else:
        pts = POLYGONS[shape]
        m = len(pts)
        side = [math.dist(pts[i], pts[(i + 1) % m]) for i in range(m)]
        cells = max(n - 2 * graded * m, 3 * m)
        cut = [int(round(cells * sum(side[:i]) / sum(side))) for i in range(m + 1)]
        ns = [max(3, b - a) for a, b in zip(cut, cut[1:])]
        t = G.polygon_graded_n(pts, ns, graded, 0.15).add_poly_basis(0).arrays()
    if degree:
        ne, nb = len(t["kind"]), degree + 1
        t["unk_elem"] = np.repeat(np.arange(ne, dtype=np.int32), nb)
        t["unk_kind"] = np.zeros(ne * nb, np.int32)
        t["unk_param"] = np.tile(np.arange(nb, dtype=np.float64), ne)
    return t


def _sweep_problems(case, seed):
    rng = np.random.default_rng(seed)
    ks = np.linspace(case["k_lo"], case["k_hi"], case["nk"]) * (1 + 0.01 * rng.uniform(-1, 1))
    ns = [int(math.ceil(10 * k * G.ELLIPSE21_PERIMETER / (2 * math.pi)))
          for k in np.linspace(case["k_lo"], case["k_hi"], case["nk"])]
    th = rng.uniform(0, 2 * math.pi)
    return ks, ns, (math.cos(th), math.sin(th))


def _wave(case, seed):
    """(wavenumber, direction) of a seed."""
    rng = np.random.default_rng(seed)
    k = case["k"] * (1 + 0.01 * rng.uniform(-1, 1))
    th = rng.uniform(0, 2 * math.pi)
    return k, (math.cos(th), math.sin(th))


def _points(case):
    """The plotting grid: [-3, 3]^2 offset so that no point meets the boundary."""
    x = np.linspace(-3.0, 3.0, case["grid"]) + 1.37e-3
    return np.ascontiguousarray(np.stack(np.meshgrid(x, x), -1).reshape(-1, 2))


# ---- prepare / run -------------------------------------------------------------
_CTX = None


def _context():
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(0)
    return _CTX


def _matrix(n, dtype=torch.complex128):
    """A device matrix in the library's column-major layout."""
    return torch.zeros((n, n), dtype=dtype, device="cuda").t()


def prepare(case, seed):
    ctx = _context()
    s = dict(case=case, ctx=ctx)
    if case["kind"] == "sweep":
        s["k"], ns, s["dir"] = _sweep_problems(case, seed)
        s["geoms"] = [capi._GeomHold(_curve_tables("ellipse", n)) for n in ns]
        s["x"] = torch.zeros(sum(ns), dtype=torch.complex128, device="cuda")
        s["out"] = list(s["x"].split(ns))  # one buffer, a view per problem
        return s
    s["k"], s["dir"] = _wave(case, seed)
    g = s["geom"] = _tables(case["shape"], case["n"], case.get("graded", 0), case.get("degree", 0))
    n = len(g["unk_elem"])
    if case["kind"] == "scatter":
        s["out"] = torch.zeros(n, dtype=torch.complex128, device="cuda")
    elif case["kind"] == "solve":
        s["A"], s["A32"] = _matrix(n), _matrix(n, torch.complex64)
        ctx.discrete_kernel_mixed(g, "combined", s["k"], s["k"], QUAD, 2.0, 1.0, out=s["A"],
                                  out32=s["A32"])
        del s["A32"]
        s["b"] = torch.zeros(n, dtype=torch.complex128, device="cuda")
        ctx.rhs(g, s["k"], s["dir"], s["k"], QUAD, out=s["b"])
        s["out"] = torch.zeros(n, dtype=torch.complex128, device="cuda")
    elif case["kind"] == "assemble":
        s["A"] = _matrix(n)
    elif case["kind"] in ("normcond", "numrange", "spectrum"):
        s["A"], s["A32"], s["M"], s["B"] = _matrix(n), _matrix(n, torch.complex64), _matrix(n), _matrix(n)
        s["bstart"] = np.arange(n + 1, dtype=np.int32)
        if case["kind"] == "numrange":
            s["theta"] = 2 * np.pi * np.arange(case["nang"]) / case["nang"]
    elif case["kind"] == "field":
        s["coef"] = ctx.scattering_solve(g, s["k"], s["dir"], s["k"], QUAD, precision="mixed")
        s["points"] = _points(case)
    elif case["kind"] == "resonance":
        s["A"] = _matrix(n)
    return s


def run(s):
    ctx, case, k = s["ctx"], s["case"], s["k"]
    kind = case["kind"]
    if kind == "sweep":
        ctx.sweep_solve(s["geoms"], k, s["dir"], k, QUAD, case["precision"], outs=s["out"])
        return s["x"]
    g = s["geom"]
    if kind == "scatter":
        return ctx.scattering_solve(g, k, s["dir"], k, QUAD, precision=case["precision"],
                                    out=s["out"])
    if kind == "solve":
        return ctx.solve(s["A"], s["b"], precision=case["precision"], out=s["out"])
    if kind == "assemble":
        return ctx.discrete_kernel(g, case["kernel"], k, k, QUAD, out=s["A"])
    if kind == "field":
        return ctx.potential(g, s["coef"], s["points"], "single", k, 0.0, QUAD)
    if kind == "resonance":
        kc = complex(k, case["kim"])
        ctx.discrete_kernel(g, "combined", kc, abs(kc), QUAD, 2.0, 1.0, out=s["A"])
        return [s["A"], ctx.singular_values(s["A"])]
    # the studies: A = Id + 2 K, its matrix in an orthonormal basis, then the question
    if case.get("precision") == "mixed":
        ctx.discrete_kernel_mixed(g, "combined", k, k, QUAD, 2.0, 1.0, out=s["A"], out32=s["A32"])
    else:
        ctx.discrete_kernel(g, "combined", k, k, QUAD, 2.0, 1.0, out=s["A"])
    ctx.eval_ident(g, QUAD, out=s["M"])
    ctx.change_basis(s["A"], s["M"], s["bstart"], out=s["B"])
    if kind == "normcond":
        norm, cond = ctx.norm_cond(s["B"], precision=case["precision"])
        return [s["B"], norm, cond]
    if kind == "numrange":
        return [s["B"], ctx.num_range_lmax(s["B"], s["theta"], tol=NR_TOL,
                                           precision=case["precision"])]
    return [s["B"], np.sort_complex(ctx.eigenvalues(s["B"]))]


# ---- work ----------------------------------------------------------------------
def _evals(n_elem):
    """Kernel evaluations of one matrix: 25 per far pair of elements, the graded
    rules for neighbours and the element itself."""
    return 25.0 * (n_elem * n_elem - 3 * n_elem) + 225.0 * 2 * n_elem + 450.0 * n_elem


def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: 100 per kernel
    evaluation (one H0, H1 pair and its geometry serves both (i, j) and (j, i)),
    8 n^3 / 3 per factorisation, 16 n^2 per matrix-vector product pair."""
    kind = case["kind"]
    if kind == "sweep":
        ns = _sweep_problems(case, 0)[1]
        return {"bytes": sum(200.0 * n for n in ns),
                "flops": sum(50.0 * _evals(n) + 8.0 * n ** 3 / 3 for n in ns)}
    n = float(case["n"])
    if kind == "scatter":
        return {"bytes": 200.0 * n, "flops": 50.0 * _evals(n) + 8.0 * n ** 3 / 3}
    if kind == "solve":
        return {"bytes": 16.0 * n * n + 32.0 * n, "flops": 8.0 * n ** 3 / 3}
    if kind == "assemble":
        nu = n * (case["degree"] + 1)
        return {"bytes": 16.0 * nu * nu + 150.0 * n, "flops": 50.0 * _evals(n)}
    if kind == "field":
        return {"bytes": 200.0 * n + 32.0 * case["grid"] ** 2,
                "flops": 100.0 * 5 * n * case["grid"] ** 2}
    if kind == "resonance":
        return {"bytes": 16.0 * n * n, "flops": 50.0 * _evals(n) + 32.0 * n ** 3 / 3}
    study = {"normcond": 8.0 * n ** 3 / 3 + 100 * 16.0 * n * n,
             "numrange": 16.0 * n * n * 15 * case.get("nang", 0),
             "spectrum": 100.0 * n ** 3 / 3}[kind]
    return {"bytes": 32.0 * n * n, "flops": 50.0 * _evals(n) + study}


# ---- exact values: the same quantities in plain torch, 64 bits -----------------
def _dev(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def _elem(g, e, t):
    """Map, normal and |J| of elements e at parameters t (tensors of one shape)."""
    p = _dev(g["param"])[e]
    kind = int(g["kind"][0])
    if kind == G.SEGMENT:
        dx, dy = p[..., 2] - p[..., 0], p[..., 3] - p[..., 1]
        x, y = p[..., 0] + dx * t, p[..., 1] + dy * t
    else:
        h = p[..., 1] - p[..., 0]
        a = p[..., 0] + h * t
        if kind == G.ELLIPSEARC:
            w = p[..., 5] - p[..., 4]
            ph = p[..., 4] + a * w
            x, y = p[..., 2] * torch.cos(ph), p[..., 3] * torch.sin(ph)
            dx, dy = -p[..., 2] * w * torch.sin(ph) * h, p[..., 3] * w * torch.cos(ph) * h
        else:
            ph, w = 2 * math.pi * a, 2 * math.pi
            c, s = torch.cos(ph), torch.sin(ph)
            if kind == G.CIRCLE:
                x, y, dx, dy = c, s, -w * s * h, w * c * h
            else:  # kite
                x, y = c + 0.65 * torch.cos(2 * ph) - 0.65, 1.5 * s
                dx, dy = (-w * s - 1.3 * w * torch.sin(2 * ph)) * h, 1.5 * w * c * h
    l = torch.sqrt(dx * dx + dy * dy)
    return x, y, dy / l, -dx / l, l


def _bessel(z):
    """J0, Y0, J1, Y1 for Re z > 0, Im z <= 0 (torch's own Bessel functions are
    off by 1e-6): power series, Miller's recurrence with Neumann's series for Y
    (Abramowitz & Stegun 9.1.10-13, 9.1.88), Hankel's expansion (9.2.5-9.2.10)."""
    out = [torch.empty_like(z) for _ in range(4)]
    r = z.abs()
    eg, tp = 0.57721566490153286061, 2 / math.pi
    for m, part in ((r < 2, 0), ((r >= 2) & (r < 25), 1), (r >= 25, 2)):
        x = z[m]
        if x.numel() == 0:
            continue
        if part == 0:
            q, lg = -x * x / 4, torch.log(x / 2)
            t, h, j0, s0, j1, s1 = torch.ones_like(x), 0.0, 1.0, 0.0, 1.0, -2 * eg + 1.0
            for n in range(1, 22):
                t, h = t * q / (n * n), h + 1.0 / n
                j0, s0 = j0 + t, s0 + t * h
                j1, s1 = j1 + t / (n + 1), s1 + t / (n + 1) * (2 * h - 2 * eg + 1.0 / (n + 1))
            j1, s1 = j1 * x / 2, s1 * x / 2
            v = (j0, tp * ((lg + eg) * j0 - s0), j1, tp * (lg * j1 - 1 / x) - s1 / math.pi)
        elif part == 1:
            hi, lo = torch.zeros_like(x), torch.full_like(x, 1e-200)
            norm, s0, s1 = (torch.zeros_like(x) for _ in range(3))
            for n in range(90, 0, -1):  # lo = J_n, hi = J_{n+1}, unnormalised
                if n % 2 == 0:
                    s0 = s0 + (-1) ** (n // 2) / (n // 2) * lo
                elif n > 1:
                    s1 = s1 + (-1) ** (n // 2) * n / ((n // 2) * (n // 2 + 1)) * lo
                if z.is_complex():  # e^{iz} = J0 + 2 sum i^n J_n: no cancellation for Im z <= 0
                    norm = norm + 2 * 1j ** n * lo
                elif n % 2 == 0:
                    norm = norm + 2 * lo
                hi, lo = lo, 2 * n / x * lo - hi
            f = (torch.exp(1j * x) if z.is_complex() else 1.0) / (norm + lo)
            j0, j1, lg = lo * f, hi * f, torch.log(x / 2)
            v = (j0, tp * ((lg + eg) * j0 - 2 * s0 * f), j1,
                 tp * ((lg + eg - 1) * j1 - j0 / x - s1 * f))
        else:
            v = []
            e = torch.sqrt(1 / (math.pi * x))
            c, s = torch.cos(x), torch.sin(x)
            for mu in (0, 4):
                t, a = torch.ones_like(x), [1.0, 0.0]  # P, Q
                for n in range(1, 31):
                    t = t * (mu - (2 * n - 1) ** 2) / (n * 8 * x)
                    a[n % 2] = a[n % 2] + (-1) ** (n // 2) * t
                # cos, sin of x - pi/4 and of x - 3 pi/4, times sqrt 2
                cc, ss = (c + s, s - c) if mu == 0 else (s - c, -s - c)
                v += [e * (a[0] * cc - a[1] * ss), e * (a[0] * ss + a[1] * cc)]
        for o, w in zip(out, v):
            o[m] = w
    return out


def _kernel(kernel, k, eta, x, y):
    """K(x, y) for test points x and trial points y, each (x, y, nx, ny, ...)."""
    wx, wy = x[0] - y[0], x[1] - y[1]
    d = torch.sqrt(wx * wx + wy * wy)
    d = torch.where(d > 0, d, torch.ones_like(d))  # coincident points belong to the graded rules
    j0, y0, j1, y1 = _bessel(k * d)
    mul = (lambda u, v: u + 1j * v) if j0.is_complex() else torch.complex
    h0, h1 = mul(j0, y0), mul(j1, y1)
    if kernel == "single":
        return 0.25j * h0
    dot = -(y[2] * wx + y[3] * wy) if kernel == "double" else x[2] * wx + x[3] * wy
    r = -0.25j * k * (dot / d) * h1
    return r + 0.25 * eta * h0 if kernel == "combined" else r


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1), 0.5 * w


def _boxes(boxes, gx, gw):
    out = []
    for a, b, c, d in boxes:
        for i in range(len(gx)):
            for j in range(len(gx)):
                out.append((a + (b - a) * gx[i], c + (d - c) * gx[j], (b - a) * (d - c) * gw[i] * gw[j]))
    return _dev(np.array(out)).T


def _rules():
    """The graded rules of an element with itself (on the square that the Duffy
    map unfolds), with its previous and with its next element."""
    L, N, sg = QUAD
    gx, gw = _gauss(N)
    xl = [sg ** (L - i) for i in range(L)] + [1.0]
    r1 = [(xl[i], xl[i + 1], xl[j], xl[j + 1]) for i in range(L) for j in range(L)]
    r2, r3 = [], []
    for l in range(L):
        a, b = sg ** (l + 1), sg ** l
        r2 += [(0, a, 1 - b, 1 - a), (a, b, 1 - b, 1 - a), (a, b, 1 - a, 1)]
        r3 += [(1 - b, 1 - a, 0, a), (1 - b, 1 - a, a, b), (1 - a, 1, a, b)]
    return _boxes(r1, gx, gw), _boxes(r2, gx, gw), _boxes(r3, gx, gw)


def _exact_matrix(g, nb, kernel, k, eta, alpha, beta):
    """beta * mass + alpha * kernel matrix on a closed curve with nb monomials
    per element."""
    ne = len(g["kind"])
    deg = torch.arange(nb, device="cuda", dtype=torch.float64)
    gx, gw = map(_dev, _gauss(QUAD[1]))
    e = torch.arange(ne, device="cuda")
    X = _elem(g, e[:, None].expand(ne, len(gx)), gx.expand(ne, len(gx)))
    F = (X[4] * gw)[..., None] * gx[:, None] ** deg  # [e, q, basis]
    A = torch.zeros((ne, nb, ne, nb), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 25) // (ne * len(gx) ** 2))
    for i in range(0, ne, step):
        x = [v[i:i + step, :, None, None] for v in X]
        K = _kernel(kernel, k, eta, x, [v[None, None] for v in X])
        Fi = F[i:i + step].to(K.dtype)
        A[i:i + step] = torch.einsum("iqjb,iqa->iajb", torch.einsum("iqjr,jrb->iqjb", K, F.to(K.dtype)), Fi)
    r1, r2, r3 = _rules()

    def block(et, ex, s, t, w):  # pairs (et, ex) with rule points (s, t, w)
        P = len(s)
        x = _elem(g, et[:, None].expand(-1, P), s.expand(len(et), P))
        y = _elem(g, ex[:, None].expand(-1, P), t.expand(len(et), P))
        K = _kernel(kernel, k, eta, x, y) * (x[4] * y[4] * w)
        bs, bt = s[:, None] ** deg, t[:, None] ** deg
        return torch.einsum("ep,pa,pb->eab", K, bs.to(K.dtype), bt.to(K.dtype))

    u, v, w = r1
    A[e, :, e, :] = (block(e, e, u, (1 - v) * u, u * w) + block(e, e, 1 - u, 1 - u + v * u, u * w))
    nx = (e + 1) % ne
    A[e, :, nx, :] = block(e, nx, *r3)
    A[nx, :, e, :] = block(nx, e, *r2)
    A *= alpha
    mass = torch.einsum("eq,q,qa,qb->eab", X[4], gw, gx[:, None] ** deg, gx[:, None] ** deg)
    if beta:
        A[e, :, e, :] += beta * mass
    return A.reshape(ne * nb, ne * nb), mass


def _exact_rhs(g, k, d):
    gx, gw = map(_dev, _gauss(QUAD[1]))
    ne = len(g["kind"])
    e = torch.arange(ne, device="cuda")
    x, y, nx, ny, l = _elem(g, e[:, None].expand(ne, len(gx)), gx.expand(ne, len(gx)))
    f = torch.exp(1j * k * (d[0] * x + d[1] * y))
    v = 1j * k * f * (nx * d[0] + ny * d[1]) - 1j * k * f
    return 2 * (v * l * gw).sum(1)


def exact(case, seed):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "sweep" or (kind in ("scatter", "solve") and n > 5000):
        return None  # minutes
    k, d = _wave(case, seed)
    nb = case.get("degree", 0) + 1
    g = _tables(case["shape"], n, case.get("graded", 0), nb - 1)
    if kind == "assemble":
        return _exact_matrix(g, nb, case["kernel"], k, k, 1.0, 0.0)[0]
    if kind == "resonance":
        kc = complex(k, case["kim"])
        A = _exact_matrix(g, 1, "combined", kc, abs(kc), 2.0, 1.0)[0]
        return [A, torch.linalg.svdvals(A)]
    A, mass = _exact_matrix(g, 1, "combined", k, k, 2.0, 1.0)
    if kind in ("scatter", "solve"):
        return torch.linalg.solve(A, _exact_rhs(g, k, d))
    if kind == "field":
        c = torch.linalg.solve(A, _exact_rhs(g, k, d))
        gx, gw = map(_dev, _gauss(QUAD[1]))
        ne = len(g["kind"])
        e = torch.arange(ne, device="cuda")
        Y = [v.reshape(-1) for v in _elem(g, e[:, None].expand(ne, len(gx)), gx.expand(ne, len(gx)))]
        w = c.repeat_interleave(len(gx)) * (Y[4] * gw.repeat(ne))
        P = _dev(_points(case))
        out = []
        for i in range(0, len(P), 4096):
            p = P[i:i + 4096]
            out.append(_kernel("single", k, 0.0, [p[:, 0:1], p[:, 1:2]], Y) @ w)
        return torch.cat(out)
    u = torch.sqrt(mass.reshape(-1))
    B = A / (u[:, None] * u)
    del A
    if kind == "spectrum":
        return [B, np.sort_complex(np.linalg.eigvals(B.cpu().numpy()))]
    if kind == "normcond":
        if n > 1500:
            return [B, None, None]
        sv = torch.linalg.svdvals(B)
        return [B, float(sv[0]), float(sv[0] / sv[-1])]
    if n > 400:
        return [B, None]
    z = torch.exp(1j * _dev(2 * np.pi * np.arange(case["nang"]) / case["nang"]))[:, None, None]
    return [B, torch.linalg.eigvalsh(0.5 * (z * B + z.conj() * B.conj().T))[:, -1]]
