"""Timed cases of this framework's work, from the smallest calls to the largest.

Five kinds, each through the package's public entry points:

* ``resolve``  — a ``Solver`` kept by the program is reset and solved again (a model solved
  again and again, a warm start, the benchmark's device-resident form);
* ``solve``    — one ``solve()`` call from host arrays to host arrays: validation, upload,
  transpose, scaling, power iteration, iterations, solution back;
* ``batch``    — a ``BatchSolver`` kept by the program solves its LPs and every solution is fetched;
* ``trait``    — the reference's host loop over the ``Backend`` methods of ``CudaBackend``;
* ``triplets`` — ``csr_from_triplets`` from host arrays to host arrays.

The LPs are the benchmark's families (random, power-law column degrees, transportation) at
the sizes of its workloads, of the tests and of the serving range (1e3 to 1e7 nonzeros, 4e7
for the single large LP). Every solve runs a fixed number of iterations (tolerance 0, as the
benchmark's timed region does), so a pass is the same work on every run.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda:0"
L2_BYTES = 126e6
CHECK = 64  # iterations between checks (SolverParams.check_every)


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # The smallest LP that anyone solves in earnest (a unit-test or a component model):
        # launches and latency are all there is. 200 x 400, 3-6 nonzeros a column.
        dict(name="resolve tiny", kind="resolve", lp="random", m=200, n=400, deg_min=3, deg_max=6, iters=1280,
             precision="fp64"),
        # A middle-sized instance of the uneven batch (m up to 2000), solved by itself; the
        # iteration limit is no multiple of the check interval.
        dict(name="resolve small", kind="resolve", lp="random", m=1417, n=2834, deg_min=3, deg_max=8, iters=1000,
             precision="fp64"),
        # A request of the serving range: 40k columns with 5 nonzeros each.
        dict(name="resolve 200k nnz", kind="resolve", lp="random", m=20_000, n=40_000, deg_min=5, deg_max=5,
             iters=640, precision="fp64"),
        # The same range's upper part in the mixed form (FP32 products, FP64 state).
        dict(name="resolve 2M nnz mixed", kind="resolve", lp="random", m=200_001, n=400_003, deg_min=3, deg_max=7,
             iters=320, precision="mixed"),
        # The transportation LP of the benchmark: 8M nonzeros, two a column, 2000 a row.
        dict(name="resolve transport", kind="resolve", lp="transport", supplies=2000, demands=2000, iters=320,
             precision="fp64"),
        # The benchmark's single large LP, FP64 and mixed: power-law column degrees.
        dict(name="resolve 40M nnz", kind="resolve", lp="powerlaw", m=2_000_000, n=4_000_000, nnz=40_000_000,
             iters=192, precision="fp64"),
        dict(name="resolve 10M nnz mixed", kind="resolve", lp="powerlaw", m=500_000, n=1_000_000, nnz=10_000_000,
             iters=192, precision="mixed"),
        # One call on a small LP: set-up counts as much as the iterations.
        dict(name="solve 3k nnz", kind="solve", lp="random", m=300, n=600, deg_min=3, deg_max=8, iters=640,
             precision="fp64"),
        # One call on the scale-test LP (200k x 400k, 3M nonzeros, power-law columns).
        dict(name="solve 3M nnz", kind="solve", lp="powerlaw", m=200_000, n=400_000, nnz=3_000_000, iters=640,
             precision="fp64"),
        # A quarter of the 4096-LP uneven batch, m log-uniform in [50, 2000]. FP64 only: the
        # batch's tuner picks each LP's summation from timings, so two processes' FP32 sums
        # differ in their rounding and could not be compared.
        dict(name="batch 1024 LPs", kind="batch", lp="batch", count=1024, m_min=50, m_max=2000, deg_min=3, deg_max=8,
             iters=640, precision="fp64"),
        # A Rust host's loop over the trait's methods on the scale-test LP: one check interval.
        dict(name="trait 3M nnz", kind="trait", lp="powerlaw", m=200_000, n=400_000, nnz=3_000_000, iters=64),
        # A model read in as triplets, with repeated entries to be summed.
        dict(name="triplets 2M", kind="triplets", m=200_000, n=400_000, count=2_000_000, repeats=0.05),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _drawn_lp(rng, nnz_lo, nnz_hi):
    """An LP of one of the three families with about log-uniform many nonzeros."""
    nnz = _log_uniform(rng, nnz_lo, nnz_hi)
    family = rng.choice(["random", "random", "powerlaw", "transport"])
    if family == "transport" or (family == "powerlaw" and nnz < 20_000):
        arcs = max(100, min(nnz // 2, 4_000_000))
        s = max(2, int(math.sqrt(arcs) * math.exp(rng.uniform(-0.7, 0.7))))
        return dict(lp="transport", supplies=s, demands=max(2, arcs // s)), 2 * arcs
    if family == "powerlaw":
        n = max(100, int(nnz / rng.uniform(6, 14)))
        return dict(lp="powerlaw", m=max(50, int(n * rng.uniform(0.3, 0.8))), n=n, nnz=nnz), nnz
    lo = rng.randint(2, 6)
    hi = lo + rng.randint(0, 6)
    n = max(30, int(2 * nnz / (lo + hi)))
    return dict(lp="random", m=max(25, int(n * rng.uniform(0.3, 0.9))), n=n, deg_min=lo, deg_max=hi), nnz


def draw(rng):
    kind = rng.choice(["resolve"] * 9 + ["solve"] * 4 + ["batch"] * 3 + ["trait"] * 2 + ["triplets"] * 2)
    prec = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "triplets":
        count = _log_uniform(rng, 1_000, 4_000_000)
        n = max(10, int(count / rng.uniform(3, 10)))
        return dict(kind=kind, m=max(10, int(n * rng.uniform(0.3, 1.5))), n=n, count=count,
                    repeats=round(rng.uniform(0.0, 0.2), 3))
    if kind == "batch":
        lo = rng.randint(20, 300)
        return dict(kind=kind, lp="batch", count=rng.randint(16, 1000), m_min=lo, m_max=rng.randint(lo + 50, 2000),
                    deg_min=rng.randint(2, 4), deg_max=rng.randint(5, 9), iters=rng.choice([100, 320, 640]),
                    precision="fp64")
    if kind == "trait":
        lp, _ = _drawn_lp(rng, 3_000, 6_000_000)
        return dict(kind=kind, **lp, iters=rng.randint(16, 96))
    lp, nnz = _drawn_lp(rng, 1_000, 16_000_000 if kind == "resolve" else 4_000_000)
    most = max(64, min(1500, int(2.5e9 / nnz)))
    return dict(kind=kind, **lp, iters=rng.randint(64, most), precision=prec)


# ------------------------------------------------------------------ inputs, from the seed alone

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _rand(shape, g):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _row_sums(rp, terms):
    """Each row's sum of its terms, the same bits on every call."""
    return torch.segment_reduce(terms, "sum", offsets=rp, initial=0.0)


def _csr(m, n, rows, cols, g):
    """A matrix with N(0,1) values at the distinct (row, column) pairs among those given."""
    key = torch.unique(rows * n + cols)
    r, c = key // n, key % n
    v = torch.randn(key.numel(), generator=g, device=DEV, dtype=torch.float64)
    rp = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(r, minlength=m), 0)
    return rp, r, c, v


def _powerlaw_degrees(n, nnz, m, g):
    """Zipf(1.5) on [2, 5000], scaled by one factor so that the total is at most nnz."""
    k = torch.arange(2, 5001, device=DEV, dtype=torch.float64)
    cdf = torch.cumsum(k ** -1.5, 0)
    d = 2.0 + torch.searchsorted(cdf, _rand(n, g) * cdf[-1]).double().clamp(max=4998)
    lo, hi = 0.0, 1.0
    for _ in range(40):
        f = 0.5 * (lo + hi)
        if float(torch.floor(d * f).clamp(min=2).sum()) <= nnz:
            lo = f
        else:
            hi = f
    return torch.floor(d * lo).clamp(min=2, max=max(2, m // 2)).long()


def _bounds(m, n, rp, c, v, half, g):
    """x0 in [0, 1]^n; rows below `half` equalities A x0, the others <= A x0 + U[0, 1]; 0 <= x <= 10."""
    x0 = _rand(n, g)
    b = _row_sums(rp, v * x0[c])
    slack = _rand(m, g)
    lc = torch.where(half, b, torch.full_like(b, -math.inf))
    uc = torch.where(half, b, b + slack)
    return lc, uc, torch.zeros(n, dtype=torch.float64, device=DEV), torch.full((n,), 10.0, dtype=torch.float64, device=DEV)


class _Lp:
    """One or more LPs side by side (block-diagonal), on the GPU: `ri`, `cj` the instance of
    each row and column, `ms`, `ns`, `zs` the instances' sizes."""


def _lp(case, seed):
    g = _gen(seed)
    p = _Lp()
    fam = case["lp"]
    if fam == "transport":
        s, d = case["supplies"], case["demands"]
        p.m, p.n = s + d, s * d
        j = torch.arange(p.n, device=DEV)
        rows = torch.stack([j // d, s + j % d])
        p.rp = torch.zeros(p.m + 1, dtype=torch.int64, device=DEV)
        p.rp[1:] = torch.cumsum(torch.bincount(rows.reshape(-1), minlength=p.m), 0)
        p.r, order = torch.sort(rows.reshape(-1), stable=True)
        p.c = torch.cat([j, j])[order]
        p.v = torch.ones(2 * p.n, dtype=torch.float64, device=DEV)
        supply = torch.floor(_rand(s, g) * 1000) + 1
        cut = torch.sort(torch.floor(_rand(d - 1, g) * (supply.sum() - d)) if d > 1 else _rand(0, g)).values
        edge = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), cut, (supply.sum() - d).reshape(1)])
        b = torch.cat([supply, edge[1:] - edge[:-1] + 1])
        p.lc, p.uc = b, b.clone()
        p.cost = torch.floor(_rand(p.n, g) * 100) + 1
        p.lv = torch.zeros(p.n, dtype=torch.float64, device=DEV)
        p.uv = torch.full((p.n,), math.inf, dtype=torch.float64, device=DEV)
        ms, ns = [p.m], [p.n]
    else:
        if fam == "batch":
            # the quantiles of the log-uniform law, in the order that requests came in
            k, lo, hi = case["count"], math.log(case["m_min"]), math.log(case["m_max"])
            ms = [int(math.exp(lo + (hi - lo) * ((37 * i) % k + 0.5) / k) + 0.5) for i in range(k)]
            ns = [2 * m for m in ms]
        else:
            ms, ns = [case["m"]], [case["n"]]
        mt, nt = torch.tensor(ms, device=DEV), torch.tensor(ns, device=DEV)
        p.m, p.n = sum(ms), sum(ns)
        m0, n0 = torch.cumsum(mt, 0) - mt, torch.cumsum(nt, 0) - nt
        cj = torch.repeat_interleave(torch.arange(len(ms), device=DEV), nt)
        if fam == "powerlaw":
            deg = _powerlaw_degrees(p.n, case["nnz"], p.m, g)
        else:
            deg = torch.randint(case["deg_min"], case["deg_max"] + 1, (p.n,), generator=g, device=DEV)
        cols = torch.repeat_interleave(torch.arange(p.n, device=DEV), deg)
        inst = cj[cols]
        rows = m0[inst] + torch.minimum((_rand(cols.numel(), g) * mt[inst]).long(), mt[inst] - 1)
        p.rp, p.r, p.c, p.v = _csr(p.m, p.n, rows, cols, g)
        ri = torch.repeat_interleave(torch.arange(len(ms), device=DEV), mt)
        half = (torch.arange(p.m, device=DEV) - m0[ri]) < mt[ri] // 2
        p.lc, p.uc, p.lv, p.uv = _bounds(p.m, p.n, p.rp, p.c, p.v, half, g)
        p.cost = 2.0 * _rand(p.n, g) - 1.0
    p.count, p.ms, p.ns = len(ms), ms, ns
    p.ri = torch.repeat_interleave(torch.arange(p.count, device=DEV), torch.tensor(ms, device=DEV))
    p.cj = torch.repeat_interleave(torch.arange(p.count, device=DEV), torch.tensor(ns, device=DEV))
    return p


def _problems(p):
    """The LPs as the package's LpProblem objects (host arrays)."""
    import saddlepoint_b200 as sp

    rp, c, v = p.rp.cpu().numpy(), p.c.int().cpu().numpy(), p.v.cpu().numpy()
    cost, lc, uc, lv, uv = (t.cpu().numpy() for t in (p.cost, p.lc, p.uc, p.lv, p.uv))
    out, i0, j0 = [], 0, 0
    for m, n in zip(p.ms, p.ns):
        i1, j1 = i0 + m, j0 + n
        a, b = int(rp[i0]), int(rp[i1])
        out.append(sp.LpProblem(m, n, rp[i0:i1 + 1] - a, c[a:b] - np.int32(j0), v[a:b].copy(), cost[j0:j1].copy(),
                                lc[i0:i1].copy(), uc[i0:i1].copy(), lv[j0:j1].copy(), uv[j0:j1].copy()))
        i0, j0 = i1, j1
    return out


def _triplets(case, seed):
    """Distinct (row, column) pairs in no order, a share of them given twice or more (to be
    summed) and one in a hundred with the value zero (to be dropped)."""
    g = _gen(seed)
    k, extra = case["count"], int(case["count"] * case["repeats"])
    cells = case["m"] * case["n"]
    key = torch.unique(torch.randint(0, cells, (3 * k,), generator=g, device=DEV))
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)[:k - extra]]
    zeros = key.numel() // 100
    again = torch.randint(zeros, key.numel(), (extra,), generator=g, device=DEV)
    # positive eighths: any order of a run's additions gives the same sum, and none is zero
    vals = torch.randint(1, 801, (key.numel() + extra,), generator=g, device=DEV).double() / 8
    vals[:zeros] = 0.0
    perm = torch.randperm(vals.numel(), generator=g, device=DEV)
    key = torch.cat([key, key[again]])[perm]
    return key // case["n"], key % case["n"], vals[perm]


def _params(case):
    import saddlepoint_b200 as sp

    return sp.SolverParams(tolerance=0.0, infeasibility_tolerance=0.0, max_iterations=case["iters"],
                           precision=sp.Precision.Mixed if case["precision"] == "mixed" else sp.Precision.FP64)


def _col_starts(p):
    trp = torch.zeros(p.n + 1, dtype=torch.int64, device=DEV)
    trp[1:] = torch.cumsum(torch.bincount(p.c, minlength=p.n), 0)
    return trp


_backend = None


def _the_backend():
    """The one backend that a program keeps open."""
    global _backend
    if _backend is None:
        import saddlepoint_b200 as sp

        _backend = sp.CudaBackend(0)
    return _backend


def _step_size(p):
    """A step size for the trait loop: 0.9 / sqrt(max row sum x max column sum of |A|)."""
    a = p.v.abs()
    rows = _row_sums(p.rp, a).max()
    cols = _row_sums(_col_starts(p), a[torch.argsort(p.c, stable=True)]).max()
    return 0.9 / math.sqrt(float(rows) * float(cols))


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    import saddlepoint_b200 as sp

    be = _the_backend()
    kind = case["kind"]
    if kind == "triplets":
        rows, cols, vals = (t.cpu().numpy() for t in _triplets(case, seed))
        return dict(kind=kind, backend=be, m=case["m"], n=case["n"], rows=rows, cols=cols, vals=vals)
    p = _lp(case, seed)
    if kind == "trait":
        lp = _problems(p)[0]
        order = torch.argsort(p.c, stable=True)
        trp = _col_starts(p)
        at = (trp.cpu().numpy(), p.r[order].int().cpu().numpy(), p.v[order].cpu().numpy())
        s = sp.ScaledProblem(p.m, p.n, (lp.row_ptr, lp.col_idx, lp.values), at, lp.c, lp.lc, lp.uc, lp.lv, lp.uv,
                             np.ones(p.m), np.ones(p.n), 1.0, 1.0)
        vec = {k: be.upload(np.zeros(n)) for k, n in
               [("x", p.n), ("xt", p.n), ("xb", p.n), ("x0", p.n), ("aty", p.n), ("tn", p.n), ("y", p.m),
                ("yt", p.m), ("y0", p.m), ("ax", p.m), ("tm", p.m), ("tm2", p.m)]}
        return dict(kind=kind, backend=be, problem=be.load(s), eta=_step_size(p), iters=case["iters"], **vec)
    lps = _problems(p)
    del p
    if kind == "batch":
        return dict(kind=kind, batch=sp.BatchSolver(lps, _params(case), be))
    if kind == "resolve":
        return dict(kind=kind, solver=sp.Solver(lps[0], _params(case), be))
    return dict(kind=kind, lp=lps[0], params=_params(case), backend=be)


def _solution(s):
    return {"x": s.x, "y": s.y, "objective": np.float64(s.objective), "dual_objective": np.float64(s.dual_objective),
            "primal_residual": np.float64(s.primal_residual), "dual_residual": np.float64(s.dual_residual),
            "norm": np.float64(s.norm_estimate), "iterations": s.iterations, "restarts": s.restarts}


def run(state):
    kind = state["kind"]
    if kind == "resolve":
        state["solver"].reset()
        return _solution(state["solver"].solve())
    if kind == "solve":
        import saddlepoint_b200 as sp

        return _solution(sp.solve(state["lp"], state["params"], state["backend"]))
    if kind == "batch":
        b = state["batch"]
        res, _ = b.solve()
        sols = [b.solution(i) for i in range(b.count)]
        out = {"x": np.concatenate([s[0] for s in sols]), "y": np.concatenate([s[1] for s in sols])}
        for k in ("objective", "dual_objective", "primal_residual", "dual_residual"):
            out[k] = np.array([getattr(r, k) for r in res])
        out["iterations"] = np.array([r.iterations for r in res])
        return out
    if kind == "triplets":
        import saddlepoint_b200 as sp

        return sp.csr_from_triplets(state["m"], state["n"], state["rows"], state["cols"], state["vals"],
                                    state["backend"])
    return _run_trait(state)


def _run_trait(s):
    """The reference's loop: PDHG iterations from zero and the statistics of one check."""
    be, p, eta = s["backend"], s["problem"], s["eta"]
    x, xt, xb, x0, aty, y, yt, y0, ax = (s[k] for k in ("x", "xt", "xb", "x0", "aty", "y", "yt", "y0", "ax"))
    be.copy(x0, x)
    be.copy(y0, y)
    for k in range(s["iters"]):
        be.spmv_t(p, y, aty)
        be.primal_step(p, x, aty, eta, xt, xb)
        be.spmv(p, xb, ax)
        be.dual_step(p, y, ax, eta, yt)
        if k + 1 < s["iters"]:
            w = (k + 1) / (k + 2)
            be.halpern_step(x, xt, x0, w, 1.0)
            be.halpern_step(y, yt, y0, w, 1.0)
    be.sub(xt, x, s["tn"])
    be.sub(yt, y, s["tm2"])
    be.spmv(p, s["tn"], s["tm"])
    res = [be.norm_sq(s["tn"]), be.norm_sq(s["tm2"]), be.dot(s["tm2"], s["tm"])]
    be.spmv(p, xt, s["tm"])
    ps = be.primal_stats(p, xt, s["tm"])
    be.spmv_t(p, yt, s["tn"])
    ds = be.dual_stats(p, yt, s["tn"])
    res += [ps.residual_sq, ps.objective, ds.residual_sq, ds.objective,
            be.step_dual_residual_sq(p, x, xt, aty, s["tn"], eta)]
    be.sub(yt, y0, s["tm"])
    be.spmv_t(p, s["tm"], s["tn"])
    d = be.dual_ray_stats(p, s["tm"], s["tn"])
    be.sub(xt, x0, s["tn"])
    be.spmv(p, s["tn"], s["tm"])
    r = be.primal_ray_stats(p, s["tn"], s["tm"])
    res += [d.objective, d.violation_sq, d.norm_sq, r.objective, r.violation_sq, r.norm_sq,
            be.distance_sq(xt, x0), be.distance_sq(yt, y0)]
    return {"x": be.download(xt), "y": be.download(yt), "scalars": [np.float64(v) for v in res]}


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Bytes and operations of one pass. An LP that fits the L2 cache (each one of a batch
    does) is read once and its iterations cost arithmetic only; a larger one's matrix (both
    layouts, 12 bytes a nonzero) and vectors cross HBM in every iteration."""
    if case["kind"] == "triplets":
        k = case["count"]
        return {"bytes": 24.0 * k + 12.0 * k + 8.0 * case["m"], "flops": float(k)}
    count = 1
    if case["lp"] == "transport":
        m, n = case["supplies"] + case["demands"], case["supplies"] * case["demands"]
        z = 2 * n
    elif case["lp"] == "powerlaw":
        m, n, z = case["m"], case["n"], case["nnz"]
    else:
        if case["lp"] == "batch":
            count = case["count"]
            lo, hi = case["m_min"], case["m_max"]
            m = (hi - lo) / math.log(hi / lo)  # the mean of the log-uniform law
            n = 2 * m
        else:
            m, n = case["m"], case["n"]
        z = n * 0.5 * (case["deg_min"] + case["deg_max"])
    vb = 8 if case.get("precision") == "mixed" else 12
    resident = 24.0 * z + 72.0 * n + 56.0 * m
    it = case["iters"]
    bytes_ = count * (12.0 * z + 32.0 * n + 24.0 * m)
    if resident > L2_BYTES:
        bytes_ += it * count * (2.0 * vb * z + 60.0 * n + 52.0 * m)
    its = it + (400 if case["kind"] == "solve" else 0)
    return {"bytes": bytes_, "flops": its * count * (4.0 * z + 12.0 * n + 12.0 * m)}


# ------------------------------------------------------------------ the same in plain torch, 64 bits

class _Segs:
    """Sums over each instance's entries; scalars of one instance broadcast."""

    def __init__(self, idx, count):
        self.idx, self.count = idx, count

    def sum(self, v):
        if self.count == 1:
            return v.sum().reshape(1)
        return torch.zeros(self.count, dtype=torch.float64, device=DEV).index_add_(0, self.idx, v)

    def of(self, t):
        return t if self.count == 1 else t[self.idx]


def _mat(rp, c, v, n):
    return torch.sparse_csr_tensor(rp, c, v, size=(rp.numel() - 1, n))


def _excess(v, lo, hi):
    return torch.where(v < lo, v - lo, torch.where(v > hi, v - hi, torch.zeros_like(v)))


def _bound_term(v, lo, hi):
    z = torch.zeros_like(v)
    up = torch.where((v > 0) & torch.isfinite(lo), v * torch.where(torch.isfinite(lo), lo, z), z)
    return torch.where((v < 0) & torch.isfinite(hi), v * torch.where(torch.isfinite(hi), hi, z), up)


def _forbidden(v, lo, hi):
    bad = ((v > 0) & (lo == -math.inf)) | ((v < 0) & (hi == math.inf))
    return torch.where(bad, v, torch.zeros_like(v))


def _recession(v, lo, hi):
    inf = torch.full_like(v, math.inf)
    z = torch.zeros_like(v)
    return _excess(v, torch.where(torch.isfinite(lo), z, -inf), torch.where(torch.isfinite(hi), z, inf))


def _clamp(v, lo, hi):
    return torch.minimum(torch.maximum(v, lo), hi)


def _inv_sqrt(v):
    ok = (v > 0) & torch.isfinite(v)
    return torch.where(ok, 1.0 / torch.sqrt(torch.where(ok, v, torch.ones_like(v))), torch.ones_like(v))


def _exact_solve(p, iters):
    r, c, v = p.r, p.c, p.v.clone()
    R, C = _Segs(p.ri, p.count), _Segs(p.cj, p.count)
    rs = torch.ones(p.m, dtype=torch.float64, device=DEV)
    cs = torch.ones(p.n, dtype=torch.float64, device=DEV)

    def ext(idx, k, how):
        t = torch.full((k,), math.inf if how == "amin" else 0.0, dtype=torch.float64, device=DEV)
        t = t.scatter_reduce_(0, idx, v.abs(), how)
        return torch.where(torch.isinf(t), torch.zeros_like(t), t)

    for _ in range(12):
        f = _inv_sqrt(ext(r, p.m, "amin") * ext(r, p.m, "amax"))
        v *= f[r]
        rs *= f
        f = _inv_sqrt(ext(c, p.n, "amin") * ext(c, p.n, "amax"))
        v *= f[c]
        cs *= f
    for k in range(11):
        if k < 10:
            fr, fc = _inv_sqrt(ext(r, p.m, "amax")), _inv_sqrt(ext(c, p.n, "amax"))
        else:
            fr = _inv_sqrt(torch.zeros_like(rs).index_add_(0, r, v.abs()))
            fc = _inv_sqrt(torch.zeros_like(cs).index_add_(0, c, v.abs()))
        v *= fr[r] * fc[c]
        rs *= fr
        cs *= fc
    cost, lc, uc, lv, uv = p.cost * cs, p.lc * rs, p.uc * rs, p.lv / cs, p.uv / cs

    def bound_norm(lo, hi):
        z = torch.zeros_like(lo)
        lo, hi = torch.where(torch.isfinite(lo), lo, z), torch.where(torch.isfinite(hi), hi, z)
        return torch.sqrt(R.sum(torch.where(lo == hi, lo * lo, lo * lo + hi * hi)))

    bs, os_ = 1.0 / (1.0 + bound_norm(lc, uc)), 1.0 / (1.0 + torch.sqrt(C.sum(cost * cost)))
    b_norm, c_norm = bound_norm(p.lc, p.uc), torch.sqrt(C.sum(p.cost * p.cost))
    lc, uc, lv, uv, cost = lc * R.of(bs), uc * R.of(bs), lv * C.of(bs), uv * C.of(bs), cost * C.of(os_)
    pf, df, of = 1.0 / (rs * R.of(bs)), 1.0 / (cs * C.of(os_)), 1.0 / (bs * os_)

    A = _mat(p.rp, c, v, p.n)
    order = torch.argsort(c, stable=True)
    trp = torch.zeros(p.n + 1, dtype=torch.int64, device=DEV)
    trp[1:] = torch.cumsum(torch.bincount(c, minlength=p.n), 0)
    AT = _mat(trp, r[order], v[order], p.m)
    del order

    # the norm of A: power iteration, each instance until its estimate settles
    j0 = torch.tensor(p.ns, device=DEV)
    local = torch.arange(p.n, device=DEV) - (torch.cumsum(j0, 0) - j0)[p.cj]
    z = 1.0 + 0.01 * (local % 7).double()
    z = z / C.of(torch.sqrt(C.sum(z * z)))
    lam = torch.zeros(p.count, dtype=torch.float64, device=DEV)
    live = torch.ones(p.count, dtype=torch.bool, device=DEV)
    for _ in range(200):
        z = AT @ (A @ z)
        norm = torch.sqrt(C.sum(z * z))
        z = z / C.of(norm)
        settled = (norm - lam).abs() <= 1e-6 * norm
        lam = torch.where(live, norm, lam)
        live &= ~settled
        if not bool(live.any()):
            break
    norm_est = torch.sqrt(lam) * 1.01
    eta = 0.998 / norm_est

    one = torch.ones(p.count, dtype=torch.float64, device=DEV)
    x, y = torch.zeros_like(cs), torch.zeros_like(rs)
    xa, ya = x.clone(), y.clone()
    omega, best_w, best_b = one.clone(), one.clone(), one * math.inf
    integral = torch.zeros_like(one)
    k, restarts = torch.zeros_like(one), torch.zeros_like(one)
    anchor, prev = one * math.inf, one * math.inf
    fresh = True
    for total in range(1, iters + 1):
        tau, sigma = eta / omega, eta * omega
        aty = AT @ y
        xt = _clamp(x - C.of(tau) * (cost - aty), lv, uv)
        ax = A @ (2.0 * xt - x)
        yt = y - R.of(sigma) * (ax - _clamp(ax - y / R.of(sigma), lc, uc))
        check = total % CHECK == 0 or total >= iters
        if check or fresh:
            dx, dy = xt - x, yt - y
            r2 = omega / eta * C.sum(dx * dx) + R.sum(dy * dy) / (eta * omega) + 2.0 * R.sum(dy * (A @ dx))
            residual = torch.sqrt(r2.clamp(min=0))
            anchor = torch.where(k == 0, residual, anchor)
            fresh = False
        w = (k + 1) / (k + 2)
        if check:
            at_t, a_t = AT @ yt, A @ xt
            e = _excess(a_t, lc, uc) * pf
            rd = cost - at_t
            f = _forbidden(rd, lv, uv) * df
            sd = (aty - at_t - (xt - x) * C.of(1.0 / tau)) * df
            pres, dres, sres = torch.sqrt(R.sum(e * e)), torch.sqrt(C.sum(f * f)), torch.sqrt(C.sum(sd * sd))
            pobj = C.sum(cost * xt) * of
            dobj = (R.sum(_bound_term(yt, lc, uc)) + C.sum(_bound_term(rd, lv, uv))) * of
        x = C.of(w) * (2.0 * xt - x) + C.of(1.0 - w) * xa
        y = R.of(w) * (2.0 * yt - y) + R.of(1.0 - w) * ya
        k = k + 1
        if not check or total >= iters:
            continue
        again = (residual <= 0.2 * anchor) | ((residual <= 0.5 * anchor) & (residual > prev)) | (k >= 0.36 * total)
        prev = residual
        # the primal weight's controller
        dxa, dya = torch.sqrt(C.sum((xt - xa) ** 2)), torch.sqrt(R.sum((yt - ya) ** 2))
        ratio = (sres / (1.0 + c_norm)) / (pres / (1.0 + b_norm))
        sane = (dxa >= 1e-16) & (dxa <= 1e12) & (dya >= 1e-16) & (dya <= 1e12) & (ratio >= 1e-8) & (ratio <= 1e8)
        err = torch.log(torch.where(sane, omega * dxa / dya, one))
        summed = 0.3 * integral + err
        new = torch.exp(torch.log(omega) - (0.99 * err + 0.01 * summed))
        balance = torch.log10(torch.where(sane, ratio, one)).abs()
        integral = torch.where(again, torch.where(sane, summed, torch.zeros_like(one)), integral)
        chosen = torch.where(sane, new, best_w)
        better = again & sane & (balance < best_b)
        best_b, best_w = torch.where(better, balance, best_b), torch.where(better, new, best_w)
        omega = torch.where(again, chosen, omega)
        restarts += again.double()
        prev = torch.where(again, one * math.inf, prev)
        k = torch.where(again, torch.zeros_like(k), k)
        ca, ra = C.of(again), R.of(again)
        x, xa = torch.where(ca, xt, x), torch.where(ca, xt, xa)
        y, ya = torch.where(ra, yt, y), torch.where(ra, yt, ya)
        fresh = True
    return dict(x=xt * cs / C.of(bs), y=yt * rs / R.of(os_), objective=pobj, dual_objective=dobj,
                primal_residual=pres, dual_residual=dres, norm=norm_est)


def _exact_trait(p, iters):
    eta = _step_size(p)
    A = _mat(p.rp, p.c, p.v, p.n)
    order = torch.argsort(p.c, stable=True)
    trp = _col_starts(p)
    AT = _mat(trp, p.r[order], p.v[order], p.m)
    x, y = torch.zeros(p.n, dtype=torch.float64, device=DEV), torch.zeros(p.m, dtype=torch.float64, device=DEV)
    for k in range(iters):
        aty = AT @ y
        xt = _clamp(x - eta * (p.cost - aty), p.lv, p.uv)
        ax = A @ (2.0 * xt - x)
        yt = y - eta * (ax - _clamp(ax - y / eta, p.lc, p.uc))
        if k + 1 < iters:
            w = (k + 1) / (k + 2)
            x, y = w * (2.0 * xt - x), w * (2.0 * yt - y)
    dx, dy = xt - x, yt - y
    axt, atyt = A @ xt, AT @ yt
    e, rd = _excess(axt, p.lc, p.uc), p.cost - atyt
    f = _forbidden(rd, p.lv, p.uv)
    sd = aty - atyt - (xt - x) / eta
    fd, fc = _forbidden(yt, p.lc, p.uc), _forbidden(-atyt, p.lv, p.uv)
    rr, rc = _recession(axt, p.lc, p.uc), _recession(xt, p.lv, p.uv)
    s = [(dx * dx).sum(), (dy * dy).sum(), (dy * (A @ dx)).sum(), (e * e).sum(), (p.cost * xt).sum(), (f * f).sum(),
         _bound_term(yt, p.lc, p.uc).sum() + _bound_term(rd, p.lv, p.uv).sum(), (sd * sd).sum(),
         _bound_term(yt, p.lc, p.uc).sum() + _bound_term(-atyt, p.lv, p.uv).sum(), (fd * fd).sum() + (fc * fc).sum(),
         (yt * yt).sum(), (p.cost * xt).sum(), (rr * rr).sum() + (rc * rc).sum(), (xt * xt).sum(), (xt * xt).sum(),
         (yt * yt).sum()]
    return {"x": xt, "y": yt, "scalars": s}


def exact(case, seed):
    if case["kind"] == "triplets":
        rows, cols, vals = _triplets(case, seed)
        key, run_of = torch.unique(rows * case["n"] + cols, return_inverse=True)
        sums = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, run_of, vals)
        return None, None, sums[sums != 0]
    p = _lp(case, seed)
    if case["kind"] == "trait":
        return _exact_trait(p, case["iters"])
    out = _exact_solve(p, case["iters"])
    if case["kind"] == "batch":
        out.pop("norm")
        return dict(out, iterations=None)
    for k in ("objective", "dual_objective", "primal_residual", "dual_residual", "norm"):
        out[k] = out[k].reshape(())
    return dict(out, iterations=None, restarts=None)
