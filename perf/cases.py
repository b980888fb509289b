"""The work this library is used for, as timed cases over its public entry
points.  Sizes are the benchmark configurations' (n = 2048 / 8192 / 16384,
batches of orders 32..512), the smoke and parity tests' (200, 777) or generic.

Every solve overwrites its matrix with the factor and its right-hand sides
with the solution, so a pass first refills both from kept copies, as the
benchmark's step does.  Matrices are column-major with the leading dimension
equal to the height (Elemental's Matrix<F> default), so odd orders arrive
with an odd leading dimension.
"""
import math

import numpy as np
import torch

import elemental_b200 as eg


def listed():
    return [
        # one small HPD system: launch and latency bound (the smoke test's order)
        {"name": "hpd_200", "op": "hpd", "n": 200, "nrhs": 3, "uplo": "lower"},
        # the plain Cholesky + solve configuration
        {"name": "hpd_2048", "op": "hpd", "n": 2048, "nrhs": 16, "uplo": "lower"},
        # an odd order, the other triangle, a single right-hand side
        {"name": "hpd_4999_upper", "op": "hpd", "n": 4999, "nrhs": 1, "uplo": "upper"},
        # the largest plain Cholesky solve (what the mixed solver is compared with)
        {"name": "hpd_16384", "op": "hpd", "n": 16384, "nrhs": 32, "uplo": "lower"},
        # GaussianElimination of a mid-size general system of odd order
        {"name": "ge_777", "op": "ge", "n": 777, "nrhs": 5},
        # the LU with partial pivoting + solve configuration
        {"name": "lu_8192", "op": "lu", "n": 8192, "nrhs": 64, "orient": "normal"},
        # the mixed-precision HPD solve configuration
        {"name": "mixed_hpd_16384", "op": "mixed_hpd", "n": 16384, "nrhs": 32, "kappa": 1e6},
        # mixed-precision GaussianElimination
        {"name": "mixed_ge_8192", "op": "mixed_ge", "n": 8192, "nrhs": 32},
        # the batched configuration, one case per kind
        {"name": "batched_hpd", "op": "batched", "kind": "hpd", "count": 4096, "nmin": 32, "nmax": 512,
         "rmin": 1, "rmax": 8, "sizes": 1},
        {"name": "batched_ge", "op": "batched", "kind": "ge", "count": 4096, "nmin": 32, "nmax": 512,
         "rmin": 1, "rmax": 8, "sizes": 2},
        # an explicit inverse (covariance / sensitivity work)
        {"name": "inverse_3000", "op": "inverse", "n": 3000},
        # a level-3 triangular solve with many right-hand sides
        {"name": "trsm_4096x3000", "op": "trsm", "m": 4096, "n": 3000, "side": "left", "uplo": "lower",
         "orient": "normal", "diag": "non_unit"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["hpd", "hpd", "ge", "lu", "mixed_hpd", "mixed_ge", "batched", "inverse", "trsm"])
    if op == "hpd":
        return {"op": op, "n": _log_int(rng, 100, 16384), "nrhs": _log_int(rng, 1, 64),
                "uplo": rng.choice(["lower", "upper"])}
    if op == "ge":
        return {"op": op, "n": _log_int(rng, 100, 8192), "nrhs": _log_int(rng, 1, 64)}
    if op == "lu":
        return {"op": op, "n": _log_int(rng, 100, 8192), "nrhs": _log_int(rng, 1, 64),
                "orient": rng.choice(["normal", "transpose"])}
    if op == "mixed_hpd":
        return {"op": op, "n": _log_int(rng, 2048, 16384), "nrhs": _log_int(rng, 1, 32),
                "kappa": 10.0 ** rng.uniform(2.0, 6.0)}
    if op == "mixed_ge":
        return {"op": op, "n": _log_int(rng, 1024, 8192), "nrhs": _log_int(rng, 1, 32)}
    if op == "batched":
        nmin = rng.randint(16, 128)
        return {"op": op, "kind": rng.choice(["hpd", "ge"]), "count": _log_int(rng, 256, 4096), "nmin": nmin,
                "nmax": rng.randint(nmin + 32, 512), "rmin": 1, "rmax": rng.randint(1, 8),
                "sizes": rng.randint(3, 1 << 20)}
    if op == "inverse":
        return {"op": op, "n": _log_int(rng, 100, 4096)}
    return {"op": "trsm", "m": _log_int(rng, 100, 4096), "n": _log_int(rng, 100, 4096),
            "side": rng.choice(["left", "right"]), "uplo": rng.choice(["lower", "upper"]),
            "orient": rng.choice(["normal", "transpose"]), "diag": rng.choice(["non_unit", "unit"])}


# ----------------------------------------------------------------- inputs --

_UPLO = {"lower": eg.LOWER, "upper": eg.UPPER}
_ORIENT = {"normal": eg.NORMAL, "transpose": eg.TRANSPOSE}
_SIDE = {"left": eg.LEFT, "right": eg.RIGHT}
_DIAG = {"non_unit": eg.NON_UNIT, "unit": eg.UNIT}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(m, n, g):
    """m x n N(0, 1), column-major."""
    return torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g).t()


def _uniform(m, n, g):
    """m x n U[-1, 1], column-major."""
    return (torch.rand(n, m, dtype=torch.float64, device="cuda", generator=g) * 2 - 1).t()


def _spd(n, g):
    """G G^T + n I, G ~ N(0, 1) (symmetric: any layout is column-major)."""
    x = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    a = x @ x.t()
    a.diagonal().add_(float(n))
    return a.t()


def _mix(x, phase):
    """A circulant orthogonal matrix (unit phases in Fourier space) times x."""
    return torch.fft.irfft(phase[:, None] * torch.fft.rfft(x, dim=0), n=x.shape[0], dim=0)


def _spd_spectrum(n, kappa, g):
    """Q diag(s) Q^T, s log-spaced over [1, kappa], Q a dense orthogonal matrix:
    the product of random circulant orthogonal matrices and permutations."""
    a = torch.diag(torch.logspace(0.0, math.log10(kappa), n, dtype=torch.float64, device="cuda"))
    perm0 = torch.randperm(n, device="cuda", generator=g)
    a = a[perm0][:, perm0]
    for _ in range(2):
        th = torch.rand(n // 2 + 1, dtype=torch.float64, device="cuda", generator=g) * (2 * math.pi)
        phase = torch.polar(torch.ones_like(th), th)
        phase[0] = 1.0
        if n % 2 == 0:
            phase[-1] = -1.0
        perm = torch.randperm(n, device="cuda", generator=g)
        a = _mix(a, phase)[perm]
        a = _mix(a.t().contiguous(), phase)[perm]
    return ((a + a.t()) * 0.5).contiguous().t()


def _sizes(case):
    r = np.random.default_rng(case["sizes"])
    n = r.integers(case["nmin"], case["nmax"] + 1, case["count"])
    k = r.integers(case["rmin"], case["rmax"] + 1, case["count"])
    return [int(x) for x in n], [int(x) for x in k]


def _offsets(sizes):
    return [0] + [int(x) for x in np.cumsum(sizes)]


def _batch(case, seed):
    """The flat arenas of A and B and the views of the systems in them."""
    g = _gen(seed)
    n, k = _sizes(case)
    offa, offb = _offsets([x * x for x in n]), _offsets([x * y for x, y in zip(n, k)])
    if case["kind"] == "hpd":
        a = torch.empty(offa[-1], dtype=torch.float64, device="cuda")
        z = torch.randn(offa[-1], dtype=torch.float64, device="cuda", generator=g)
        for i, x in enumerate(n):
            gi = z[offa[i]:offa[i + 1]].view(x, x)
            ai = a[offa[i]:offa[i + 1]].view(x, x)
            torch.mm(gi, gi.t(), out=ai)
            ai.diagonal().add_(float(x))
    else:
        a = torch.rand(offa[-1], dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    b = torch.randn(offb[-1], dtype=torch.float64, device="cuda", generator=g)
    return n, k, offa, offb, a, b


def _triangle(case, g):
    """A triangular factor as a solver has it: the Cholesky factor of an HPD
    matrix (unit: its columns divided by the diagonal, the diagonal arbitrary
    and never read)."""
    nt = case["m"] if case["side"] == "left" else case["n"]
    f = torch.linalg.cholesky(_spd(nt, g))
    if case["diag"] == "unit":
        f = f / f.diagonal()[None, :]
        f.diagonal().fill_(3.0)
    f = f.contiguous()  # row-major lower = column-major upper
    return f if case["uplo"] == "upper" else f.t().contiguous()


def _inputs(case, seed):
    """(A, B) of one call, column-major."""
    g = _gen(seed)
    op = case["op"]
    if op == "hpd":
        return _spd(case["n"], g), _normal(case["n"], case["nrhs"], g)
    if op in ("ge", "lu", "mixed_ge"):
        return _uniform(case["n"], case["n"], g), _normal(case["n"], case["nrhs"], g)
    if op == "mixed_hpd":
        return _spd_spectrum(case["n"], case["kappa"], g), _normal(case["n"], case["nrhs"], g)
    if op == "inverse":
        return _uniform(case["n"], case["n"], g), None
    return _triangle(case, g).t(), _normal(case["m"], case["n"], g)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    s.h = eg.Handle(0)
    if case["op"] == "batched":
        n, k, offa, offb, s.a0, s.b0 = _batch(case, seed)
        s.a, s.b = s.a0.clone(), s.b0.clone()
        va = [torch.as_strided(s.a, (x, x), (1, x), offa[i]) for i, x in enumerate(n)]
        vb = [torch.as_strided(s.b, (x, y), (1, x), offb[i]) for i, (x, y) in enumerate(zip(n, k))]
        s.plan = eg.BatchPlan(s.h, 0 if case["kind"] == "hpd" else 1, va, vb)
        return s
    s.a0, s.b0 = _inputs(case, seed)
    s.a = s.a0.clone()
    s.b = None if s.b0 is None else s.b0.clone()
    if case["op"] == "lu":
        s.p = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
    return s


def run(s):
    case = s.case
    op = case["op"]
    if op == "mixed_hpd":
        return s.h.hpd_solve_mixed(s.a0, s.b0)[0]
    if op == "mixed_ge":
        return s.h.gaussian_elimination_mixed(s.a0, s.b0)[0]
    if op == "trsm":
        s.b.copy_(s.b0)
        s.h.trsm(_SIDE[case["side"]], _UPLO[case["uplo"]], _ORIENT[case["orient"]], _DIAG[case["diag"]], 1.0, s.a0,
                 s.b)
        return s.b
    s.a.copy_(s.a0)
    if op == "inverse":
        s.h.inverse(s.a)
        return s.a
    s.b.copy_(s.b0)
    if op == "hpd":
        s.h.hpd_solve(s.a, s.b, uplo=_UPLO[case["uplo"]])
        return s.a, s.b
    if op == "ge":
        s.h.gaussian_elimination(s.a, s.b)
        return s.a, s.b
    if op == "lu":
        s.h.lu(s.a, s.p)
        s.h.lu_solve_after(s.a, s.p, s.b, orient=_ORIENT[case["orient"]])
        return s.a, s.p, s.b
    s.plan.run()
    return s.a, s.b


def work(case):
    """Inputs read once, outputs written once, and the textbook flops."""
    op = case["op"]
    if op == "batched":
        n, k = _sizes(case)
        w = 1.0 / 3.0 if case["kind"] == "hpd" else 2.0 / 3.0
        f = 1.0 if case["kind"] == "ge" else 0.5  # the share of A that is referenced
        return {"bytes": float(sum(16 * (f * x * x + x * y) for x, y in zip(n, k))),
                "flops": float(sum(w * x ** 3 + 2.0 * x * x * y for x, y in zip(n, k)))}
    if op == "trsm":
        m, n = case["m"], case["n"]
        nt = m if case["side"] == "left" else n
        return {"bytes": 4.0 * nt * nt + 16.0 * m * n, "flops": 1.0 * m * n * nt}
    n = float(case["n"])
    if op == "inverse":
        return {"bytes": 16.0 * n * n, "flops": 2.0 * n ** 3}
    k = case["nrhs"]
    if op == "hpd":
        return {"bytes": 8.0 * n * n + 16.0 * n * k, "flops": n ** 3 / 3 + 2 * n * n * k}
    if op == "mixed_hpd":
        return {"bytes": 4.0 * n * n + 16.0 * n * k, "flops": n ** 3 / 3 + 2 * n * n * k}
    b = 8.0 if op == "mixed_ge" else 16.0
    return {"bytes": b * n * n + 16.0 * n * k, "flops": 2 * n ** 3 / 3 + 2 * n * n * k}


def exact(case, seed):
    op = case["op"]
    if op == "batched":
        n, k, offa, offb, a, b = _batch(case, seed)
        hpd = case["kind"] == "hpd"
        for i, (x, y) in enumerate(zip(n, k)):
            m = a[offa[i]:offa[i + 1]].view(x, x).t()
            r = b[offb[i]:offb[i + 1]].view(y, x).t()
            if hpd:
                f = torch.linalg.cholesky(m)
                r.copy_(torch.cholesky_solve(r, f))
                m.copy_(torch.tril(f) + torch.triu(m, 1))
            else:
                r.copy_(torch.linalg.solve(m, r))
        return (a if hpd else None), b
    a, b = _inputs(case, seed)
    if op == "hpd":
        f = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(b, f)
        f = torch.tril(f) + torch.triu(a, 1) if case["uplo"] == "lower" else torch.triu(f.t()) + torch.tril(a, -1)
        return f, x
    if op in ("mixed_hpd", "mixed_ge"):
        if op == "mixed_hpd":
            f = torch.linalg.cholesky(a)
            solve = lambda r: torch.cholesky_solve(r, f)  # noqa: E731
        else:
            lu, piv = torch.linalg.lu_factor(a)
            solve = lambda r: torch.linalg.lu_solve(lu, piv, r)  # noqa: E731
        x = solve(b)
        return x + solve(b - a @ x)
    if op == "ge":
        return None, torch.linalg.solve(a, b)  # the eliminated A has no textbook form below the diagonal
    if op == "lu":
        lu, piv = torch.linalg.lu_factor(a)
        x = torch.linalg.lu_solve(lu, piv, b, adjoint=case["orient"] == "transpose")
        return lu, None, x
    if op == "inverse":
        return torch.linalg.inv(a)
    t = torch.tril(a) if case["uplo"] == "lower" else torch.triu(a)
    if case["diag"] == "unit":
        t = t - torch.diag(t.diagonal()) + torch.eye(t.shape[0], dtype=t.dtype, device=t.device)
    if case["orient"] == "transpose":
        t = t.t()
    up = (case["uplo"] == "upper") != (case["orient"] == "transpose")
    return torch.linalg.solve_triangular(t, b, upper=up, left=case["side"] == "left")
