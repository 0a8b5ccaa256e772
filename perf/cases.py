"""The calls this library is used for, as timed cases.

A case is a dict of plain values.  ``listed()`` gives the fixed cases,
``draw(rng)`` one more from the same ranges.  ``prepare(case, seed)`` builds
what a program holds before the call, ``run(state)`` makes the call through
the package's public entry points and returns its outputs, ``work(case)``
gives the bytes and operations a call cannot do without, and
``exact(case, seed)`` the outputs as plain torch computes them in 64 bits.

Kinds of cases:
  track   -- DeviceTracker.run: paths of a homotopy from start to end points
  eval    -- DeviceBatch.evaldiff: values and gradients at power series
  bals    -- DeviceBals.solve: block-Toeplitz least squares
  newton  -- DeviceNewton.solve: Newton's method on power series
  diag    -- endgame.series_diagnostics_device: diagnostics at points of paths

Operation counts use the multiple-double weights of the reference
(double-double add 20, multiply 23; quad-double add 89, multiply 336; a
complex product four real ones and a complex sum two).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from phcpack_b200 import benchwork, dense, endgame, homotopy, newton, series, trackwork, workloads

ADD = {1: 1, 2: 20, 4: 89}
MUL = {1: 1, 2: 23, 4: 336}
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest tracking job: all roots of one small system, one call
        dict(name="track_small", kind="track", form="dense", n=4, paths=16, systems=1, pmode=1, rmode=2, learned=False),
        # the benchmark's batch: 1024 paths, double predictor, learned step
        dict(name="track_1024", kind="track", form="dense", n=10, paths=1024, systems=1, pmode=1, rmode=2,
             learned=True),
        # many systems of mixed sizes in one batch, most paths diverging, end points refined in quad-double
        dict(name="track_mixed_qd", kind="track", form="sparse", n=14, paths=2048, systems=16, pmode=1, rmode=4,
             learned=False),
        # all in double-double, polynomials of degree 3 (products of three variables)
        dict(name="track_dd_cubic", kind="track", form="cubic", n=5, paths=243, systems=1, pmode=2, rmode=2,
             learned=False),
        # one system at one vector of series: a single evaluation inside a user's own loop
        dict(name="eval_one", kind="eval", systems=1, n=8, deg=15, nmon=12, maxvar=4, expmax=2, prec=2, cplx=True),
        # the benchmark's systems: n = 32, degree 31, complex double-double
        dict(name="eval_dd_1024", kind="eval", systems=1024, n=32, deg=31, nmon=32, maxvar=4, expmax=3, prec=2,
             cplx=True),
        # quad-double at an odd degree and dimension, products of up to seven variables
        dict(name="eval_qd", kind="eval", systems=48, n=17, deg=20, nmon=12, maxvar=7, expmax=1, prec=4, cplx=False),
        # long series (degree 95)
        dict(name="eval_dd_deg95", kind="eval", systems=32, n=16, deg=95, nmon=16, maxvar=4, expmax=2, prec=2,
             cplx=False),
        # the benchmark's least squares: 64 x 64 quad-double blocks, degree 31
        dict(name="bals_qd_512", kind="bals", inst=512, n=64, deg=31, tile=32, prec=4, cplx=False),
        # complex double-double, a dimension off the powers of two
        dict(name="bals_dd_cplx", kind="bals", inst=200, n=24, deg=16, tile=8, prec=2, cplx=True),
        # Newton's method on one system, four steps from the start series
        dict(name="newton_one", kind="newton", systems=1, n=8, deg=15, nmon=4, maxvar=3, prec=2, cplx=False, steps=4),
        # end-game diagnostics at a batch of points
        dict(name="diag_1024", kind="diag", n=10, paths=1024, pmode=2),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["track", "track", "eval", "eval", "eval", "bals", "bals", "newton", "diag"])
    if kind == "track":
        form = rng.choice(["dense", "dense", "sparse", "cubic"])
        pmode = rng.choice([1, 1, 2]) if form != "sparse" else 1
        if form == "cubic":
            n = rng.randint(2, 5)
            paths = _logint(rng, 1, 3 ** n)
        else:
            n = rng.randint(3, 11 if form == "sparse" else 10)
            paths = _logint(rng, 1, min(2 ** n, 1024 if pmode == 1 else 200))
        return dict(kind="track", form=form, n=n, paths=paths, systems=1, pmode=pmode,
                    rmode=rng.choice([2, 2, 4]), learned=pmode == 1 and rng.random() < 0.5)
    if kind == "eval":
        prec, cplx = rng.choice([1, 2, 2, 4]), rng.random() < 0.5
        deg = rng.randint(1, 31) if rng.random() < 0.75 else rng.randint(32, 110)
        n = _logint(rng, 2, 32)
        maxvar = rng.randint(1, min(n, 6))
        nmon = _logint(rng, 2, 32)
        cost = n * nmon * 3 * maxvar * (deg + 1) ** 2 / 2 * (MUL[prec] + ADD[prec]) * (4 if cplx else 1)
        cap = max(1, min(1024, int(4e10 / cost)))
        return dict(kind="eval", systems=_logint(rng, 1, cap), n=n, deg=deg, nmon=nmon, maxvar=maxvar,
                    expmax=rng.randint(1, 3), prec=prec, cplx=cplx)
    if kind == "bals":
        prec, cplx = rng.choice([1, 2, 2, 4, 4]), rng.random() < 0.4
        tile = rng.choice([3, 4, 8, 10, 16, 32])
        n = tile * rng.randint(1, max(1, 64 // tile))
        if cplx and prec == 4:
            n = min(n, tile * max(1, 40 // tile))
        deg = rng.randint(1, 31)
        cost = (8 / 3 * n ** 3 + deg * deg / 2 * n * n) * (MUL[prec] + ADD[prec]) * (4 if cplx else 1)
        cap = max(1, min(512, int(2e11 / cost)))
        return dict(kind="bals", inst=_logint(rng, 1, cap), n=n, deg=deg, tile=tile, prec=prec, cplx=cplx)
    if kind == "newton":
        n = rng.randint(2, 16)
        return dict(kind="newton", systems=_logint(rng, 1, 64), n=n, deg=rng.randint(3, 24), nmon=rng.randint(2, 6),
                    maxvar=min(3, n), prec=rng.choice([2, 2, 4]), cplx=rng.random() < 0.5, steps=rng.randint(2, 5))
    n = rng.randint(2, 10)
    return dict(kind="diag", n=n, paths=_logint(rng, 1, min(2 ** n, 1024)), pmode=rng.choice([1, 2, 2]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _limbs(hi, prec, g):
    """prec-limb numbers with the leading limbs hi and random lower limbs."""
    parts = [hi]
    for _ in range(prec - 1):
        parts.append(parts[-1] * 2.0 ** -53 * (torch.rand(hi.shape, generator=g, device=DEV, dtype=torch.float64)
                                               * 2 - 1))
    for i in range(prec - 1, 0, -1):
        s = parts[i - 1] + parts[i]
        parts[i - 1], parts[i] = s, parts[i] - (s - parts[i - 1])
    return torch.stack(parts, dim=-1)


def _numbers(shape, prec, cplx, kind, g, scale=None):
    f64 = dict(generator=g, device=DEV, dtype=torch.float64)
    if kind == "unit" and cplx:
        th = torch.rand(shape, **f64) * (2 * math.pi)
        parts = [torch.cos(th), torch.sin(th)]
    else:
        parts = [torch.randn(shape, **f64) if kind == "normal" else torch.rand(shape, **f64) * 2 - 1
                 for _ in range(2 if cplx else 1)]
    if scale is not None:
        parts = [p * scale for p in parts]
    return torch.cat([_limbs(p, prec, g) for p in parts], dim=-1).reshape(-1)


def _supports(rng, nsys, n, nmon, maxvar, expmax):
    """nmon monomials per polynomial over up to maxvar distinct variables, as
    workloads.random_supports draws them, built array-wise."""
    total = nsys * n * nmon
    nvr = rng.integers(1, maxvar + 1, size=total).astype(np.int32)
    pick = np.argsort(rng.random((total, n)), axis=1)[:, :maxvar]
    used = np.arange(maxvar)[None, :] < nvr[:, None]
    idx = np.where(used, np.sort(np.where(used, pick, n), axis=1), 0).astype(np.int32)
    exps = np.where(used, rng.integers(1, expmax + 1, size=(total, maxvar)), 0).astype(np.int32)
    return np.arange(0, total + 1, nmon, dtype=np.int32), nvr, idx, exps


def _eval_batch(c, seed):
    g = _gen(seed)
    n1 = c["deg"] + 1
    total = c["systems"] * c["n"]
    off, nvr, idx, exps = _supports(np.random.default_rng(seed), c["systems"], c["n"], c["nmon"], c["maxvar"],
                                    c["expmax"])
    kind = "unit" if c["cplx"] else "uniform"
    cff = _numbers((len(nvr), n1), c["prec"], c["cplx"], kind, g)
    cst = _numbers((total, n1), c["prec"], c["cplx"], kind, g)
    # series decaying as 2^-k, as the package's workloads draw them
    scale = 2.0 ** -torch.arange(n1, device=DEV, dtype=torch.float64)
    inp = _numbers((total, n1), c["prec"], c["cplx"], "normal", g, scale)
    return workloads.SystemBatch(c["systems"], c["n"], c["deg"], c["maxvar"], c["prec"], c["cplx"], off, nvr, idx,
                                 exps, cst.cpu().numpy(), cff.cpu().numpy(), inp.cpu().numpy())


def _bals_inputs(c, seed):
    g = _gen(seed)
    n1, n = c["deg"] + 1, c["n"]
    scale = None
    if c["cplx"]:  # Jacobian series inside their radius of convergence
        scale = (2.0 ** -torch.arange(n1, device=DEV, dtype=torch.float64)).view(1, n1, 1, 1)
    mat = _numbers((c["inst"], n1, n, n), c["prec"], c["cplx"], "normal", g, scale)
    rhs = _numbers((c["inst"], n1, n), c["prec"], c["cplx"], "normal", g, None if scale is None else scale[..., 0])
    return mat, rhs


def _newton_batch(c, seed):
    """Systems with the known power-series solution x_i(t) = e_i (1 + t/2 +
    t^2/4 + ...), the constants chosen so that f(x) = 0 holds at degree 0 and
    the start series the solution truncated there."""
    rng = np.random.default_rng(seed)
    nsys, n, n1, prec, cplx = c["systems"], c["n"], c["deg"] + 1, c["prec"], c["cplx"]
    # polynomial i: a multiple of x_i, then products over other variables
    nvr, idx, off = [], [], [0]
    for _ in range(nsys):
        for i in range(n):
            sups = [(i,)] + [tuple(sorted(rng.choice(n, int(rng.integers(1, c["maxvar"] + 1)), replace=False)))
                             for _ in range(c["nmon"] - 1)]
            for sup in sups:
                nvr.append(len(sup))
                idx.append(list(sup) + [0] * (c["maxvar"] - len(sup)))
            off.append(len(nvr))
    nvr, idx, off = np.array(nvr, np.int32), np.array(idx, np.int32), np.array(off, np.int32)
    exps = (np.arange(c["maxvar"])[None, :] < nvr[:, None]).astype(np.int32)
    W = prec * (2 if cplx else 1)
    # short dyadic values, so that the constant coefficients are exact
    x0 = rng.integers(4, 12, size=(nsys, n)) / 8.0
    cf = np.zeros((len(nvr), n1, W))
    lead = rng.integers(-8, 9, size=len(nvr)) / 16.0
    lead[off[:-1]] = 4.0
    cf[:, 0, 0] = lead
    if n1 > 1:
        cf[:, 1, 0] = rng.integers(-8, 9, size=len(nvr)) / 16.0
    cst = np.zeros((nsys * n, n1, W))
    for p in range(nsys * n):
        s = p // n
        cst[p, 0, 0] = -sum(cf[m, 0, 0] * np.prod(x0[s, idx[m, :nvr[m]]]) for m in range(off[p], off[p + 1]))
    start = np.zeros((nsys * n, n1, W))
    start[:, 0, 0] = x0.reshape(-1)
    return workloads.SystemBatch(nsys, n, c["deg"], c["maxvar"], prec, cplx, off, nvr, idx, exps, cst.reshape(-1),
                                 cf.reshape(-1), start.reshape(-1))


def _cubic(rng, n):
    """Degree-3 polynomials: a cube, products of up to three variables and
    lower terms, unit-circle coefficients."""
    polys = []
    for i in range(n):
        mons = {((i, 3),), (), ((i, 1),)}
        for _ in range(5):
            vs = sorted(rng.choice(n, min(n, 3), replace=False).tolist())
            mons.add(tuple((v, 1) for v in vs))
            j, k = sorted(rng.choice(n, 2, replace=True).tolist())
            mons.add(((j, 2),) if j == k else ((j, 1), (k, 1)))
        mons = sorted(mons)
        polys.append([(m, complex(z)) for m, z in zip(mons, homotopy.unit(rng, len(mons)))])
    return polys


def _track_problem(c, seed):
    rng = np.random.default_rng(seed)
    if c["form"] == "dense":
        targets, maxvar = [homotopy.dense_quadratic(rng, c["n"]) for _ in range(c["systems"])], 2
    elif c["form"] == "cubic":
        targets, maxvar = [_cubic(rng, c["n"]) for _ in range(c["systems"])], 3
    else:
        lo = min(6, c["n"])
        sizes = [c["n"]] + [int(rng.integers(lo, c["n"] + 1)) for _ in range(c["systems"] - 1)]
        targets, maxvar = [homotopy.sparse_quadratic(rng, n) for n in sizes], 2
    return homotopy.total_degree_problem(targets, complex(homotopy.unit(rng)),
                                         max_paths_per_system=max(1, c["paths"] // c["systems"]), rng=rng,
                                         maxvar=maxvar)


def prepare(case, seed):
    c = case
    if c["kind"] == "track":
        dt = homotopy.DeviceTracker(_track_problem(c, seed))
        if c["learned"]:
            dt.set_model(trackwork.load_model_bytes())
        return dict(kind="track", dt=dt, args=dict(pmode=c["pmode"], rmode=c["rmode"], step_mode=int(c["learned"])))
    if c["kind"] == "eval":
        return dict(kind="eval", batch=series.DeviceBatch(_eval_batch(c, seed)))
    if c["kind"] == "bals":
        d = dense.DeviceBals(c["prec"], c["cplx"], c["inst"], c["n"], c["deg"] + 1, c["tile"])
        mat, rhs = _bals_inputs(c, seed)
        d.mat.copy_(mat)
        return dict(kind="bals", solver=d, rhs=rhs)
    if c["kind"] == "newton":
        return dict(kind="newton", solver=newton.DeviceNewton(_newton_batch(c, seed)), steps=c["steps"])
    rng = np.random.default_rng(seed)
    pb = homotopy.total_degree_problem([homotopy.dense_quadratic(rng, c["n"])], complex(homotopy.unit(rng)),
                                       max_paths_per_system=c["paths"], rng=rng)
    dt = homotopy.DeviceTracker(pb)
    # the diagnostics at the start points, which lie on the paths at t = 0
    tpt = torch.zeros(pb.npaths, dtype=torch.float64, device=DEV)
    return dict(kind="diag", dt=dt, xpt=dt.arr["x0"], tpt=tpt, pmode=c["pmode"])


def run(state):
    s = state
    if s["kind"] == "track":
        dt = s["dt"]
        dt.run(**s["args"])
        return dt.xend, dt.info, dt.dinfo
    if s["kind"] == "eval":
        return s["batch"].evaldiff()
    if s["kind"] == "bals":
        # the solve overwrites the right hand sides
        d = s["solver"]
        d.rhs.copy_(s["rhs"])
        d.reset_flags()
        d.solve()
        return d.sol, d.rhs, d.Q, d.R, d.flags
    if s["kind"] == "newton":
        d = s["solver"]
        d.solve(s["steps"], torch.cuda.current_stream())
        return d.series, d.flags
    return endgame.series_diagnostics_device(s["dt"], s["xpt"], s["tpt"], pmode=s["pmode"])


# ------------------------------------------------------------------ work
def _evals(c):
    """(coefficient products, bytes) of one evaluation of a case's systems:
    monomials of (maxvar + 1) / 2 variables on average."""
    k = (c["maxvar"] + 1) / 2
    convs = max(1.0, 3 * k - 3) + k * (c.get("expmax", 1) - 1) / 2
    n1 = c["deg"] + 1
    total = c["systems"] * c["n"] * c["nmon"]
    W = 8 * c["prec"] * (2 if c["cplx"] else 1)
    nbytes = W * n1 * (total + c["systems"] * c["n"] * 2 + c["systems"] * c["n"] * (c["n"] + 1))
    return total * convs * n1 * (n1 + 1) / 2, nbytes


def _ma(prec, cplx):
    return (4 if cplx else 1) * (MUL[prec] + ADD[prec])


def work(case):
    c = case
    if c["kind"] == "eval":
        prods, nbytes = _evals(c)
        return {"bytes": nbytes, "flops": prods * _ma(c["prec"], c["cplx"])}
    if c["kind"] == "bals":
        n, d = c["n"], c["deg"]
        ma = 8 / 3 * n ** 3 + d * (d + 1) / 2 * n * n + 1.5 * (d + 1) * n * n
        W = 8 * c["prec"] * (2 if c["cplx"] else 1)
        nbytes = c["inst"] * W * ((d + 1) * n * n + 3 * (d + 1) * n + 2 * n * n)
        return {"bytes": nbytes, "flops": c["inst"] * ma * _ma(c["prec"], c["cplx"])}
    if c["kind"] == "newton":
        prods, nbytes = _evals(c)
        n, d = c["n"], c["deg"]
        ma = prods + c["systems"] * (8 / 3 * n ** 3 + d * (d + 1) / 2 * n * n + 1.5 * (d + 1) * n * n)
        return {"bytes": nbytes, "flops": c["steps"] * ma * _ma(c["prec"], c["cplx"])}
    # tracking and diagnostics: the Taylor series of a path to degree 8 and a
    # few point evaluations per step, about 20 steps per path
    n = c["n"]
    nterm = {"dense": (n + 1) * (n + 2) // 2, "sparse": 6, "cubic": 13}[c.get("form", "dense")]
    per = n * nterm * 18 + n ** 3 * (5 / 3) + 8 * n * n
    paths = c["paths"]
    if c["kind"] == "diag":
        return {"bytes": paths * (16 * n + 100), "flops": paths * (per * _ma(c["pmode"], True) + 40 * n ** 4 * 8)}
    steps = 20
    return {"bytes": paths * (16 * n + 128 * n + 40),
            "flops": paths * steps * (per * _ma(c["pmode"], True) + 2 * n * nterm * _ma(2, True))}


# ------------------------------------------------------------------ 64-bit results
def _leading(x, prec, cplx):
    """Flat limbs -> leading values (float64 or complex128)."""
    W = prec * (2 if cplx else 1)
    a = x.reshape(-1, W)
    re = a[:, :prec].sum(dim=1)
    return torch.complex(re, a[:, prec:].sum(dim=1)) if cplx else re


def _flat(x, prec, cplx):
    """float64 or complex128 values -> flat limbs with zero lower limbs."""
    parts = [x.real, x.imag] if cplx else [x]
    out = torch.zeros(x.numel(), prec * len(parts), dtype=torch.float64, device=x.device)
    for i, p in enumerate(parts):
        out[:, i * prec] = p.reshape(-1)
    return out.reshape(-1)


def _conv(a, b):
    """Truncated products of series (last dimension)."""
    n1 = a.shape[-1]
    out = torch.zeros_like(a)
    for i in range(n1):
        out[..., i:] += a[..., i:i + 1] * b[..., :n1 - i]
    return out


def _evaldiff(c, cst, cff, X, idx, exps):
    """Values (row n) and gradients of the case's systems, one row of series
    per polynomial, from the leading values of its arrays."""
    n, n1, nmon, mv = c["n"], c["deg"] + 1, c["nmon"], c["maxvar"]
    out = torch.zeros(c["systems"] * n, n + 1, n1, dtype=cff.dtype, device=DEV)
    one = torch.zeros(n1, dtype=cff.dtype, device=DEV)
    one[0] = 1
    step = max(1, (1 << 16) // (n * nmon))
    for s0 in range(0, c["systems"], step):
        s1 = min(c["systems"], s0 + step)
        m = slice(s0 * n * nmon, s1 * n * nmon)
        poly = torch.arange(s0 * n, s1 * n, device=DEV).repeat_interleave(nmon)
        sysof = poly // n
        powers, lower = [], []
        for v in range(mv):
            x, e = X[sysof * n + idx[m, v]], exps[m, v]
            low = one.expand(len(poly), n1).clone()      # x^(e-1), 1 where unused
            full = low.clone()
            for r in range(1, c.get("expmax", 1) + 1):
                nxt = _conv(full, x)
                low = torch.where((e == r).unsqueeze(1), full, low)
                full = torch.where((e >= r).unsqueeze(1), nxt, full)
            powers.append(full)
            lower.append(low)
        val = cff[m]
        for v in range(mv):
            val = _conv(val, powers[v])
        flat = out.view(-1, n1)
        flat.index_add_(0, poly * (n + 1) + n, val)
        for v in range(mv):
            d = _conv(cff[m], lower[v]) * exps[m, v].unsqueeze(1)
            for u in range(mv):
                if u != v:
                    d = _conv(d, powers[u])
            flat.index_add_(0, poly * (n + 1) + idx[m, v], d)  # exponent 0 where unused: adds zero
    out[:, n] += cst
    return out


def _eval_arrays(c, b):
    to = lambda a: torch.from_numpy(a).to(DEV)
    lead = lambda a: _leading(to(a), c["prec"], c["cplx"]).reshape(-1, c["deg"] + 1)
    return lead(b.cst), lead(b.cff), lead(b.input), to(b.idx).long(), to(b.exps).long()


def _exact_eval(c, seed):
    return _flat(_evaldiff(c, *_eval_arrays(c, _eval_batch(c, seed))), c["prec"], c["cplx"])


def _exact_newton(c, seed):
    """Newton steps on the whole series; the package leaves out updates of
    coefficients that have converged, which are zero to rounding here."""
    cst, cff, X, idx, exps = _eval_arrays(c, _newton_batch(c, seed))
    ns, n, n1 = c["systems"], c["n"], c["deg"] + 1
    for _ in range(c["steps"]):
        out = _evaldiff(c, cst, cff, X, idx, exps).view(ns, n, n + 1, n1)
        J, b = out[:, :, :n], -out[:, :, n].clone()
        lu = torch.linalg.lu_factor(J[..., 0].contiguous())
        dx = torch.zeros_like(b)
        for k in range(n1):
            dx[..., k] = torch.linalg.lu_solve(*lu, b[..., k:k + 1].contiguous()).squeeze(-1)
            b[..., k + 1:] -= torch.einsum("sijk,sj->sik", J[..., 1:n1 - k], dx[..., k])
        X = X + dx.reshape(ns * n, n1)
    return [_flat(X, c["prec"], c["cplx"]), None]


def _householder(A):
    """Q and R of the package's reflectors: the diagonal of R takes the phase
    of the entry it replaces in complex arithmetic and is nonnegative in real
    arithmetic; the last column of a square matrix is not reflected in the
    real case."""
    ni, n = A.shape[0], A.shape[1]
    R = A.clone()
    Q = torch.eye(n, dtype=A.dtype, device=A.device).expand(ni, n, n).clone()
    for k in range(n - 1):
        x = R[:, k:, k]
        x0 = x[:, 0]
        nrm = torch.linalg.vector_norm(x, dim=1)
        ph = x0 / x0.abs() if A.is_complex() else torch.ones_like(x0)
        tail2 = (x[:, 1:].abs() ** 2).sum(dim=1)
        v = x.clone()
        # x0 - ph |x|, without cancellation
        v[:, 0] = -ph * tail2 / (x0.abs() + nrm) if A.is_complex() else \
            torch.where(x0 > 0, -tail2 / (x0 + nrm), x0 - nrm)
        beta = 2.0 / (v.abs() ** 2).sum(dim=1)
        w = torch.einsum("bi,bij->bj", v.conj(), R[:, k:, :]) * beta[:, None]
        R[:, k:, :] -= v[:, :, None] * w[:, None, :]
        u = torch.einsum("bij,bj->bi", Q[:, :, k:], v) * beta[:, None]
        Q[:, :, k:] -= u[:, :, None] * v.conj()[:, None, :]
    return Q, torch.triu(R)


def _exact_bals(c, seed):
    mat, rhs = _bals_inputs(c, seed)
    n1, n, prec, cplx = c["deg"] + 1, c["n"], c["prec"], c["cplx"]
    A = _leading(mat, prec, cplx).reshape(c["inst"], n1, n, n)
    b = _leading(rhs, prec, cplx).reshape(c["inst"], n1, n).clone()
    Q, R = _householder(A[:, 0])
    x = torch.zeros_like(b)
    for k in range(n1):
        y = torch.einsum("bji,bj->bi", Q.conj(), b[:, k])
        x[:, k] = torch.linalg.solve_triangular(R, y.unsqueeze(-1), upper=True).squeeze(-1)
        if k + 1 < n1:
            b[:, k + 1:] -= torch.einsum("bkij,bj->bki", A[:, 1:n1 - k], x[:, k])
    return [_flat(v, prec, cplx) for v in (x, b, Q, R)] + [None]


def exact(case, seed):
    """None for tracking and diagnostics: their results follow from step
    decisions that plain 64-bit arithmetic does not restate."""
    if case["kind"] == "eval":
        return _exact_eval(case, seed)
    if case["kind"] == "bals":
        return _exact_bals(case, seed)
    if case["kind"] == "newton":
        return _exact_newton(case, seed)
    return None
