"""The work a user of this library has it do, as measurable cases: factorizations, refactorizations and solves through the
public entry points, over the range of sizes, matrix families, value types, right-hand-side counts and options they are
used at.  ``listed()`` names the fixed cases, ``draw(rng)`` gives another of the same ranges, ``prepare`` makes what a
program has in hand before the call (the matrix, its analysis, the factors or the captured graph), ``run`` is one pass.

Matrix families (values from the seed, as in ``fplus_b200.workloads``):

* ``band``      one spectral pencil: a complex band with a few dense tau rows and columns
* ``pencil``    the coupled pencil of a spectral solver (Fourier modes x fields x Chebyshev modes, dense tau lines)
* ``stencil2d`` / ``stencil3d``   nonsymmetric convection-diffusion on a square or cubic grid, real
* ``random``    a random complex pattern with row and column scales over 8 decades each
"""
import ctypes
import math
import random

import numpy as np
import torch

import fplus_b200 as F
from fplus_b200 import workloads as W

PRECISION = {"fp64": F.PREC_FP64, "fp32": F.PREC_FP32, "bf16x3": F.PREC_BF16X3, "tf32": F.PREC_TF32}


def listed():
    return [
        # the smallest call: one right-hand side of a 1-D spectral problem, once per time step, factors on the device
        dict(name="solve_band_n900", do="solve", family="band", n=900, hbw=5, ntau=3, nrhs=1, trans=0),
        # a 1-D pencil refactored and solved from host buffers when the time step changes
        dict(name="step_band_n2500", do="factor", family="band", n=2500, hbw=7, ntau=2, nrhs=1, trans=0, host=True),
        # the 100 x 100 stencil, host buffers in and out: the drop-in use of fplus_factor + fplus_solve
        dict(name="step_stencil2d_g100", do="factor", family="stencil2d", g=100, nrhs=1, trans=0, host=True),
        # a larger 2-D grid of odd size, values and right-hand side on the device
        dict(name="step_stencil2d_g401", do="factor", family="stencil2d", g=401, nrhs=1, trans=0, host=False),
        # the shift-invert pencil of the headline benchmark: refactorization and one solve
        dict(name="step_pencil_n32768", do="factor", family="pencil", modes=8, fields=4, nc=1024, nrhs=1, trans=0, host=False),
        # the same pencil's solve alone: what an eigenvalue iteration repeats on one factorization
        dict(name="solve_pencil_n32768", do="solve", family="pencil", modes=8, fields=4, nc=1024, nrhs=1, trans=0),
        # adjoint solves of a mid-size pencil of odd sizes, several right-hand sides
        dict(name="adjoint_pencil_n4995", do="solve", family="pencil", modes=5, fields=3, nc=333, nrhs=12, trans=2),
        # a block of right-hand sides against one 3-D factorization
        dict(name="solve_stencil3d_g40_r32", do="solve", family="stencil3d", g=40, nrhs=32, trans=0),
        # a 3-D grid in FP64: large fronts, the Schur updates dominate
        dict(name="step_stencil3d_g48", do="factor", family="stencil3d", g=48, nrhs=1, trans=0, host=False),
        # the precision form on a larger 3-D grid: reduced-precision Schur updates, refined to FP64 accuracy
        dict(name="mixed_stencil3d_g56", do="factor", family="stencil3d", g=56, nrhs=1, trans=0, host=False, precision="bf16x3"),
        # nearly dense factors (complex, badly scaled) and many right-hand sides
        dict(name="step_random_n9001_r48", do="factor", family="random", n=9001, nrhs=48, trans=0, host=False),
        # many uneven pencils refactored and solved as one CUDA graph, values and right-hand sides from the host
        dict(name="batch_band_48", do="batch", family="band", count=48, nmin=500, nmax=4000, nrhs=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    family = rng.choice(["band", "pencil", "pencil", "stencil2d", "stencil3d", "random", "batch"])
    if family == "batch":
        return dict(do="batch", family="band", count=rng.randint(8, 48), nmin=rng.randint(300, 700), nmax=_log(rng, 1000, 4000),
                    nrhs=rng.randint(1, 8))
    do = rng.choice(["factor", "solve"])
    c = dict(do=do, family=family, nrhs=rng.choice([1, 1, _log(rng, 2, 48)]), trans=rng.choice([0, 0, 1, 2]))
    if do == "factor":
        c["host"] = rng.random() < 0.4
    if family == "band":
        c.update(n=_log(rng, 300, 8000), hbw=rng.randint(4, 8), ntau=rng.randint(2, 4))
    elif family == "pencil":
        fields = rng.randint(2, 4)
        modes = rng.randint(1, 8)
        c.update(modes=modes, fields=fields, nc=_log(rng, 48, 1024))
    elif family == "stencil2d":
        c.update(g=_log(rng, 16, 400))
    elif family == "stencil3d":
        c.update(g=_log(rng, 8, 46))
        if do == "factor" and rng.random() < 0.4:
            c["precision"] = rng.choice(["fp32", "bf16x3", "tf32"])
    else:
        c.update(n=_log(rng, 500, 8500))
    return c


def _phases(rng, m, lo, hi):
    return 10.0 ** rng.uniform(np.log10(lo), np.log10(hi), m) * np.exp(1j * rng.uniform(0.0, 2.0 * np.pi, m))


def _csc(n, rows, cols, vals):
    key = cols * n + rows
    _, first = np.unique(key, return_index=True)
    rows, cols, vals = rows[first], cols[first], vals[first]
    Ap = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int64)
    return n, Ap, np.ascontiguousarray(rows, np.int64), np.ascontiguousarray(vals)


def _band(n, hbw, ntau, seed):
    """A complex band with ntau dense rows and columns, magnitudes log-uniform in [1e-2, 1e2]."""
    rng = np.random.default_rng(seed)
    k = np.arange(n, dtype=np.int64)
    rows = np.concatenate([k[(k + d >= 0) & (k + d < n)] for d in range(-hbw, hbw + 1)])
    cols = np.concatenate([k[(k + d >= 0) & (k + d < n)] + d for d in range(-hbw, hbw + 1)])
    # the dense lines are those of boundary conditions: the last rows and columns
    taus = n - 1 - np.arange(ntau, dtype=np.int64)
    rows = np.concatenate([rows, np.repeat(taus, n), np.tile(k, ntau)])
    cols = np.concatenate([cols, np.tile(k, ntau), np.repeat(taus, n)])
    return _csc(n, rows, cols, _phases(rng, len(rows), 1e-2, 1e2))


def _random(n, seed, per_col=12):
    """A random complex pattern with a dominant diagonal, rows and columns scaled over 8 decades each; and the column scales."""
    rng = np.random.default_rng(seed)
    cols = np.concatenate([np.arange(n, dtype=np.int64), np.repeat(np.arange(n, dtype=np.int64), per_col - 1)])
    rows = np.concatenate([np.arange(n, dtype=np.int64), rng.integers(0, n, n * (per_col - 1), dtype=np.int64)])
    vals = np.exp(1j * rng.uniform(0.0, 2.0 * np.pi, len(rows)))
    vals[:n] *= per_col
    dr, dc = 10.0 ** rng.uniform(-4, 4, n), 10.0 ** rng.uniform(-4, 4, n)
    return _csc(n, rows, cols, dr[rows] * vals * dc[cols]), dc


def _matrix(case, seed):
    """(n, Ap, Ai, Ax) and the size of each unknown (None: all alike)."""
    f = case["family"]
    if f == "band":
        return _band(case["n"], case["hbw"], case["ntau"], seed), None
    if f == "pencil":
        return W.pencil(modes=case["modes"], fields=case["fields"], nc=case["nc"], lo=1e-3, hi=1e3, seed=seed), None
    if f == "stencil2d":
        return W.convdiff2d(case["g"], seed), None
    if f == "stencil3d":
        return W.convdiff3d(case["g"], seed), None
    m, dc = _random(case["n"], seed)
    return m, 1.0 / dc


def _solution(n, nrhs, cplx, size, seed):
    """The solutions the right-hand sides are made for, (n, nrhs)."""
    rng = np.random.default_rng(seed + 77)
    x = rng.standard_normal((n, nrhs))
    if cplx:
        x = x + 1j * rng.standard_normal((n, nrhs))
    return x if size is None else x * size[:, None]


def _times(matrix, x, trans):
    """op(A) x in 64 bits."""
    n, Ap, Ai, Ax = matrix
    cols = np.repeat(np.arange(n), np.diff(Ap))
    v = Ax.conj() if trans == 2 else Ax
    out = np.empty(x.shape, x.dtype)
    to, frm = (Ai, cols) if trans == 0 else (cols, Ai)
    for r in range(x.shape[1]):
        t = v * x[frm, r]
        out[:, r] = np.bincount(to, t.real, n)
        if np.iscomplexobj(t):
            out[:, r] += 1j * np.bincount(to, t.imag, n)
    return out


def _batch_sizes(case):
    """The sizes and shapes of a batch's pencils, log-uniform between its limits (the same for every seed)."""
    rng = random.Random(case["count"] * 10007 + case["nmin"])
    return [(_log(rng, case["nmin"], case["nmax"]), rng.randint(4, 8), rng.randint(2, 4)) for _ in range(case["count"])]


def _system(case, seed):
    m, size = _matrix(case, seed)
    x = _solution(m[0], case["nrhs"], np.iscomplexobj(m[3]), size, seed)
    return m, _times(m, x, case["trans"]), x


def _host_x(case):
    return case.get("host") or case.get("precision", "fp64") != "fp64"


def prepare(case, seed):
    s = dict(case, stream=torch.cuda.Stream())
    F.lib().fplus_b200_use_stream(None)
    if case["do"] == "batch":
        mats = [_band(n, hbw, ntau, seed * 1000 + k) for k, (n, hbw, ntau) in enumerate(_batch_sizes(case))]
        s["Ax"] = [m[3] for m in mats]
        s["b"] = [_times(m, _solution(m[0], case["nrhs"], True, None, seed * 1000 + k), 0) for k, m in enumerate(mats)]
        nums = F.factor_batch([F.analyze(m[0], m[1], m[2]) for m in mats], s["Ax"])
        s["graph"] = F.BatchGraph(nums, case["nrhs"])
        return s
    m, b, _ = _system(case, seed)
    s["sym"] = sym = F.analyze(m[0], m[1], m[2])
    num = sym.factor(m[3])              # the pattern's first factorization: later ones know where its dense chain starts
    if case["do"] == "solve":
        s["num"] = num
    # (the refining solve takes host right-hand sides)
    s["b"] = b if _host_x(case) else torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    s["Ax"] = m[3] if case.get("host") else torch.from_numpy(m[3]).cuda()
    torch.cuda.synchronize()
    return s


def _on(stream):
    F.lib().fplus_b200_use_stream(ctypes.c_void_p(stream.cuda_stream))


def run(s):
    if s["do"] == "batch":
        g, st = s["graph"], s["stream"]
        for k, a in enumerate(s["Ax"]):
            g.upload(k, a, s["b"][k])
        g.launch(st.cuda_stream)
        codes = g.status()
        return dict(codes=codes, x=np.concatenate([g.download(k).ravel(order="F") for k in range(len(codes))]))
    with torch.cuda.stream(s["stream"]):
        _on(s["stream"])
        if s["do"] == "solve":
            return dict(x=s["num"].solve_device(s["b"].clone(), s["trans"]))
        prec = PRECISION[s.get("precision", "fp64")]
        num = s["sym"].factor(s["Ax"], device=not s["host"], precision=prec)
        if prec:
            x, _, _ = num.solve_refine(s["b"], s["trans"])
            return dict(x=x, Dr=num.Dr, Dc=num.Dc)
        x = num.solve(s["b"], s["trans"]) if s["host"] else num.solve_device(s["b"].clone(), s["trans"])
        return dict(x=x, p=num.p, Dr=num.Dr, Dc=num.Dc)


def _factor_size(case):
    """(factor entries, complex or real multiply-adds of the elimination, entries of A, n) of one matrix."""
    f = case["family"]
    if f in ("band", "pencil"):
        # the dense lines fill U; each pivot eliminates the rows its band and the dense rows bring
        if f == "band":
            n, w, per = case["n"], 2 * case["hbw"] + case["ntau"], 2 * case["hbw"] + 1 + 2 * case["ntau"]
        else:
            n = case["modes"] * case["fields"] * case["nc"]
            w, per = (2 * 6 + 2) * case["fields"], 13 * case["fields"] + 4 * case["fields"]
        return n * n / 2 + n * w, w * n * n / 2, per * n, n
    n, Ap, Ai, Ax = _matrix(case, 1)[0]
    P = F.analyze(n, Ap, Ai).plan()
    nc, nr, npiv = np.diff(P["col_ptr"]).astype(float), P["nrows"].astype(float), np.bincount(P["col_front"], minlength=len(P["nrows"])).astype(float)
    npiv = np.minimum(npiv, nr)
    m, c = nr - npiv, nc - npiv
    return (float((nr * npiv + npiv * c).sum()), float((npiv ** 3 / 3 + npiv ** 2 / 2 * (m + c) + npiv * m * c).sum()),
            float(len(Ai)), n)


def work(case):
    if case["do"] == "batch":
        parts = [work(dict(case, do="factor", n=n, hbw=h, ntau=t)) for n, h, t in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    entries, madds, nnz, n = _factor_size(case)
    real = case["family"].startswith("stencil")
    vs, fl, nrhs = (8, 2, case["nrhs"]) if real else (16, 8, case["nrhs"])
    solve = dict(bytes=vs * (entries + 2 * n * nrhs), flops=fl * entries * nrhs)
    if case["do"] == "solve":
        return solve
    # values in, factors written once and read once by the solve
    return dict(bytes=vs * (nnz + entries) + solve["bytes"], flops=fl * madds + solve["flops"])


def exact(case, seed):
    """The solutions the right-hand sides were made for."""
    if case["do"] == "batch":
        xs = [_solution(n, case["nrhs"], True, None, seed * 1000 + k).ravel(order="F") for k, (n, _, _) in enumerate(_batch_sizes(case))]
        return dict(codes=None, x=np.concatenate(xs))
    x = _system(case, seed)[2]
    out = dict(x=x if _host_x(case) else np.ascontiguousarray(x.T))
    if case["do"] == "factor":
        out.update(Dr=None, Dc=None)
        if case.get("precision", "fp64") == "fp64":
            out.update(p=None)
    return out
