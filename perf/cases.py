"""The work that users of ganit_v2_b200 have it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program has in hand
before the call (models, resident problems, layers), ``run`` is one call
through the public API, ``work`` what that call cannot do without and
``exact`` the 64-bit answer where one is known (the solves to a tolerance
have none: the point that they stop at is the method's own).

Kinds
  oneshot   ``solve_pdhg_gpu(lp)``: model in host memory, solution back
  lp        ``Problem.solve`` on a resident random LP
  blend     ``Problem.solve`` on a resident multi-period blending LP
  qp        ``Problem.solve`` on a resident portfolio QP (diagonal-plus-low-rank Hessian)
  batch     ``BatchSolver.solve``: many LPs of uneven size
  diff      ``DiffSolver.forward`` and ``backward``
  branch    ``strong_branch``: both children of a node's candidate columns
  backend   one check period of a host program that drives the ``Backend`` operations
"""
import numpy as np
import torch

import ganit_v2_b200 as gb
from ganit_v2_b200 import workloads as W

PRECISION = {"double": gb.Precision.Double, "mixed": gb.Precision.Mixed, "dynamic": gb.Precision.Dynamic}
MAX_ITER = 40_000  # no solve here runs longer, whatever the seed


def listed():
    return [
        # the smallest call: a model of 50 rows solved once, as a service does per request
        {"name": "oneshot_small", "kind": "oneshot", "source": "random", "m": 50, "n": 125, "k_min": 6, "k_max": 6,
         "precision": "double", "tol": 1e-4},
        # a mid-size model (a year of weekly blending plans) solved once from host arrays
        {"name": "oneshot_blend_weekly", "kind": "oneshot", "source": "blend", "crudes": 60, "products": 16, "specs": 5,
         "periods": 52, "precision": "double", "tol": 1e-4},
        # the reference configuration: random LP of 40K nonzeros, the default options
        {"name": "lp_2000x5000_double", "kind": "lp", "m": 2000, "n": 5000, "k_min": 8, "k_max": 8,
         "precision": "double", "tol": 1e-4},
        # a smaller, ragged LP re-solved to a tight tolerance (FP32 phase, then FP64)
        {"name": "lp_701x1753_mixed_1e-6", "kind": "lp", "m": 701, "n": 1753, "k_min": 4, "k_max": 12,
         "precision": "mixed", "tol": 1e-6},
        # the headline: a year of daily blending plans, 2.9M nonzeros
        {"name": "blend_daily_mixed", "kind": "blend", "crudes": 60, "products": 16, "specs": 5, "periods": 365,
         "precision": "mixed", "tol": 1e-4},
        # many independent LPs at once (scenario analysis): 512 of uneven size, and a few dozen in FP64
        {"name": "batch_512_mixed", "kind": "batch", "count": 512, "m_min": 50, "m_max": 4000, "precision": "mixed",
         "tol": 1e-4},
        {"name": "batch_37_double", "kind": "batch", "count": 37, "m_min": 30, "m_max": 1500, "precision": "double",
         "tol": 1e-4},
        # portfolio optimisation: the large universe in FP64 (the default) and a desk-size one, mixed
        {"name": "qp_100000x50_double", "kind": "qp", "assets": 100_000, "factors": 50, "precision": "double",
         "tol": 1e-4},
        {"name": "qp_8009x33_mixed", "kind": "qp", "assets": 8009, "factors": 33, "precision": "mixed", "tol": 1e-4},
        # a training step through the differentiable LP layer: solutions and all gradients
        {"name": "diff_48_500x1000", "kind": "diff", "count": 48, "m": 500, "n": 1000, "k": 10, "precision": "mixed",
         "tol": 1e-6},
        # one branching decision of a MILP solver: 32 candidate columns, 64 child LPs
        {"name": "branch_5000x200", "kind": "branch", "n": 5000, "knapsacks": 200, "density": 0.02, "candidates": 32,
         "precision": "mixed", "tol": 1e-6},
        # a host program (the reference's own driver loop) on the Backend operations, FP32
        {"name": "backend_4000x10000_f32", "kind": "backend", "m": 4000, "n": 10000, "k_min": 8, "k_max": 8,
         "mat": "f32", "vec": "f32", "iterations": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["oneshot", "oneshot", "lp", "lp", "blend", "batch", "batch", "qp", "qp", "diff", "branch",
                       "backend"])
    precision = rng.choice(["double", "mixed"])
    if kind in ("oneshot", "lp"):
        tight = kind == "lp" and rng.random() < 0.4
        m = _log_int(rng, 50, 1000 if tight else 4000)
        k_min = rng.randint(4, 8)
        c = {"kind": kind, "m": m, "n": int(round(m * rng.uniform(2.0, 3.0))), "k_min": k_min,
             "k_max": k_min + rng.randint(0, 6), "precision": precision, "tol": 1e-6 if tight else 1e-4}
        if kind == "oneshot":
            c["source"] = "random"
        return c
    if kind == "blend":
        return {"kind": kind, "crudes": rng.randint(10, 60), "products": rng.randint(4, 16), "specs": rng.randint(2, 5),
                "periods": _log_int(rng, 10, 365), "precision": precision, "tol": 1e-4}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 256), "m_min": rng.randint(20, 60),
                "m_max": _log_int(rng, 200, 4000), "precision": precision, "tol": 1e-4}
    if kind == "qp":
        return {"kind": kind, "assets": _log_int(rng, 1000, 100_000), "factors": rng.randint(5, 50),
                "precision": precision, "tol": 1e-4}
    if kind == "diff":
        m = _log_int(rng, 60, 500)
        return {"kind": kind, "count": rng.randint(6, 48), "m": m, "n": 2 * m + rng.randint(0, 9), "k": rng.randint(6, 10),
                "precision": "mixed", "tol": 1e-6}
    if kind == "branch":
        n = _log_int(rng, 400, 5000)
        return {"kind": kind, "n": n, "knapsacks": max(8, n // rng.randint(20, 40)), "density": 0.02 if n > 1500 else 0.1,
                "candidates": rng.randint(4, 32), "precision": "mixed", "tol": 1e-6}
    m = _log_int(rng, 100, 4000)
    mat, vec = rng.choice([("f32", "f32"), ("f32", "f64"), ("f64", "f64")])
    return {"kind": kind, "m": m, "n": int(round(m * rng.uniform(2.0, 3.0))), "k_min": 4, "k_max": rng.randint(4, 12),
            "mat": mat, "vec": vec, "iterations": 64}


# ---------------------------------------------------------------- models
def _random_lp(case, seed):
    rng = np.random.default_rng([seed, 1])
    k = rng.integers(case["k_min"], case["k_max"] + 1, size=case["n"])
    return W.random_feasible_lp(case["m"], case["n"], np.minimum(k, case["m"]), seed=seed)


def _model(case, seed):
    if case["kind"] == "qp":
        return W.portfolio_qp(case["assets"], case["factors"], seed=seed)
    if case["kind"] == "blend" or case.get("source") == "blend":
        return W.blending_lp(case["crudes"], case["products"], case["specs"], case["periods"], seed=seed)
    if case["kind"] == "branch":
        return W.milp_node(n=case["n"], knapsacks=case["knapsacks"], density=case["density"], up_blocked=0,
                           down_blocked=0, seed=seed % (1 << 31))
    return _random_lp(case, seed)


def _models(case, seed):
    first = (seed * 1_000_003) % (1 << 40)  # no instance shared with the neighbouring seeds
    if case["kind"] == "diff":
        return W.diff_batch(case["count"], case["m"], case["n"], case["k"], seed=first)
    sizes = np.random.default_rng([case["count"], case["m_min"], case["m_max"]])  # the case's, whatever the seed
    out = []
    for i in range(case["count"]):
        m = int(round(float(np.exp(sizes.uniform(np.log(case["m_min"]), np.log(case["m_max"]))))))
        n = int(round(2.5 * m))
        k = np.minimum(sizes.integers(4, 13, size=n), m)
        out.append(W.random_feasible_lp(m, n, k, seed=first + i))
    return out


def _options(case):
    return gb.Options(tol=case["tol"], max_iter=MAX_ITER, precision=PRECISION[case["precision"]])


def _adjoints(lps, seed):
    rng = np.random.default_rng([seed, 2])
    return rng.standard_normal(sum(lp.n for lp in lps)), rng.standard_normal(sum(lp.m for lp in lps))


def _steps(lp):
    """Step sizes of a backend program: tau sigma |A|^2 < 1 from |A|^2 <= |A|_1 |A|_inf."""
    a = np.abs(lp.A.val)
    one = np.bincount(lp.A.idx, a, minlength=lp.n).max()
    inf = np.add.reduceat(np.append(a, 0.0), np.minimum(lp.A.ptr[:-1], lp.A.nnz))[np.diff(lp.A.ptr) > 0].max()
    eta = 0.99 / float(np.sqrt(one * inf))
    return 4.0 * eta, eta / 4.0


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "oneshot":
        return {"kind": kind, "lp": _model(case, seed), "opt": _options(case)}
    if kind in ("lp", "blend", "qp"):
        opt = _options(case)
        return {"kind": kind, "problem": gb.Problem(_model(case, seed), opt), "opt": opt}
    if kind == "batch":
        opt = _options(case)
        return {"kind": kind, "solver": gb.BatchSolver(_models(case, seed), opt), "opt": opt}
    if kind == "diff":
        opt = _options(case)
        lps = _models(case, seed)
        wx, wy = _adjoints(lps, seed)
        return {"kind": kind, "layer": gb.DiffSolver(lps, opt, tail_iters=200, ckpt_every=20), "opt": opt, "wx": wx,
                "wy": wy}
    if kind == "branch":
        lp = _model(case, seed)
        node = gb.solve_pdhg_gpu(lp, gb.Options(tol=1e-7, max_iter=MAX_ITER))
        cands = gb.most_fractional(node.x, gb.fractional(node.x, lp.is_int), case["candidates"])
        return {"kind": kind, "lp": lp, "x": node.x, "y": node.y, "z": node.pobj, "cands": cands, "opt": _options(case)}
    lp = _random_lp(case, seed)
    data = dict(A=lp.A, AT=lp.A.transpose(), c=lp.c, l=lp.l, u=lp.u, lo=lp.lo, hi=lp.hi, Rres=np.ones(lp.m),
                Cres=np.ones(lp.n))
    be = gb.Backend(data, case["mat"], case["vec"])
    tau, sigma = _steps(lp)
    n, m = lp.n, lp.m
    v = {k: be.zeros(n) for k in ("x0", "x", "xn", "xbar", "aty", "sumx")}
    v.update({k: be.zeros(m) for k in ("y0", "y", "yn", "ax", "sumy")})
    return {"kind": kind, "be": be, "v": v, "tau": tau, "sigma": sigma, "iterations": case["iterations"]}


def _solution(r):
    return {"x": r.x, "y": r.y, "pobj": r.pobj, "status": int(r.status)}


def _backend_period(s):
    """PDHG iterations from (x0, y0) and the KKT pieces of the last iterate."""
    be, v = s["be"], s["v"]
    be.copy(v["x0"], v["x"])
    be.copy(v["y0"], v["y"])
    be.fill(v["sumx"], 0.0)
    be.fill(v["sumy"], 0.0)
    x, xn, y, yn = v["x"], v["xn"], v["y"], v["yn"]
    for _ in range(s["iterations"]):
        be.spmv_AT(y, v["aty"])
        be.primal_step(x, v["aty"], None, s["tau"], xn, v["xbar"], v["sumx"])
        be.spmv_A(v["xbar"], v["ax"])
        be.dual_step(y, v["ax"], s["sigma"], yn, v["sumy"])
        x, xn, y, yn = xn, x, yn, y
    be.spmv_A(x, v["ax"])
    be.spmv_AT(y, v["aty"])
    rd2, vobj = be.dual_res(v["aty"])
    return {"x": x.to_host(), "y": y.to_host(), "sumx": v["sumx"].to_host(), "sumy": v["sumy"].to_host(),
            "rp2": be.primal_res2(v["ax"]), "rd2": rd2, "vobj": vobj, "robj": be.row_dual_obj(y), "cx": be.dot_c(x),
            "step2": be.diff2(x, xn)}


def run(state):
    kind = state["kind"]
    if kind == "oneshot":
        return _solution(gb.solve_pdhg_gpu(state["lp"], state["opt"]))
    if kind in ("lp", "blend", "qp"):
        return _solution(state["problem"].solve(state["opt"]))
    if kind == "batch":
        res = state["solver"].solve(state["opt"])
        return {"x": np.concatenate([r.x for r in res]), "y": np.concatenate([r.y for r in res]),
                "pobj": np.array([r.pobj for r in res]), "status": np.array([int(r.status) for r in res])}
    if kind == "diff":
        res, x, y = state["layer"].forward(state["opt"])
        g = state["layer"].backward(state["wx"], state["wy"])
        return {"x": x, "y": y, "c": g["c"], "lo": g["lo"], "hi": g["hi"], "a_val": g["a_val"],
                "pobj": np.array([r.pobj for r in res]), "status": np.array([int(r.status) for r in res])}
    if kind == "branch":
        r = gb.strong_branch(state["lp"], state["x"], state["cands"], state["z"], opt=state["opt"], y=state["y"])
        return {"z": r.z, "cert": r.cert, "status": r.status, "action": r.action, "var": r.var, "lo": r.lo, "hi": r.hi}
    return _backend_period(state)


# ---------------------------------------------------------------- work
def _size(case):
    """(nonzeros, columns, rows) of a case's models together, as the generators draw them on average."""
    kind = case["kind"]
    if kind == "qp":
        return case["assets"], case["assets"], 1
    if kind == "blend" or case.get("source") == "blend":
        c, p, s, t = case["crudes"], case["products"], case["specs"], case["periods"]
        return t * (c * p * (3 + s) + 3 * c + 3 * p), t * (c * (2 + p) + 2 * p), t * (1 + c + p + p * s)
    if kind == "batch":
        lo, hi = case["m_min"], case["m_max"]
        m = case["count"] * (hi - lo) / np.log(hi / lo)  # mean of the log-uniform size
        return 20.0 * m, 2.5 * m, m
    if kind == "diff":
        return case["count"] * case["n"] * case["k"], case["count"] * case["n"], case["count"] * case["m"]
    if kind == "branch":
        return case["n"] * case["knapsacks"] * case["density"], case["n"], case["knapsacks"]
    return case["n"] * (case["k_min"] + case["k_max"]) / 2, case["n"], case["m"]


def work(case):
    """The model read once (indices, values, vectors), the solution written once, and the
    arithmetic of one check period: 64 iterations of two products with the matrix (four with
    the factors of a QP's Hessian), whatever number of periods the tolerance takes."""
    nnz, n, m = (float(v) for v in _size(case))
    periods = 2.0 * case["candidates"] if case["kind"] == "branch" else 1.0
    nbytes = 12 * nnz + 4 * (m + 1) + 8 * (3 * n + 2 * m) + 8 * (n + m)
    flops = 64 * periods * (4 * nnz + 8 * n + 8 * m)
    if case["kind"] == "qp":
        nbytes += 8 * n * (case["factors"] + 1)
        flops += 64 * 4 * n * case["factors"]
    if case["kind"] == "diff":
        nbytes += 8 * (nnz + n + 2 * m) + 8 * (n + m)
        flops += 200 * 8 * nnz
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- exact answers
def _exact_backend(case, seed):
    lp = _random_lp(case, seed)
    tau, sigma = _steps(lp)
    rows = torch.from_numpy(np.repeat(np.arange(lp.m), np.diff(lp.A.ptr)))
    cols = torch.from_numpy(lp.A.idx.astype(np.int64))
    val = torch.from_numpy(lp.A.val)
    c, l, u, lo, hi = (torch.from_numpy(getattr(lp, k)) for k in ("c", "l", "u", "lo", "hi"))
    x, y = torch.zeros(lp.n, dtype=torch.float64), torch.zeros(lp.m, dtype=torch.float64)
    sx, sy, xp = torch.zeros_like(x), torch.zeros_like(y), x

    def mul(v):
        return torch.zeros(lp.m, dtype=torch.float64).index_add_(0, rows, val * v[cols])

    def mul_t(v):
        return torch.zeros(lp.n, dtype=torch.float64).index_add_(0, cols, val * v[rows])

    for _ in range(case["iterations"]):
        xp = x
        x = torch.minimum(torch.maximum(xp - tau * (c - mul_t(y)), l), u)
        q = y - sigma * mul(2.0 * x - xp)
        y = q + torch.minimum(torch.maximum(-q, sigma * lo), sigma * hi)
        sx, sy = sx + x, sy + y
    ax, z = mul(x), c - mul_t(y)
    p = torch.minimum(torch.maximum(ax, lo), hi)
    vobj = float((torch.clamp(z, min=0) * l + torch.clamp(z, max=0) * u).sum())  # every column here is boxed
    yl, yu = y > 0, y < 0
    robj = float((y * lo)[yl & torch.isfinite(lo)].sum() + (y * hi)[yu & torch.isfinite(hi)].sum())
    return {"x": x, "y": y, "sumx": sx, "sumy": sy, "rp2": float(((ax - p) ** 2).sum()), "rd2": None, "vobj": vobj,
            "robj": robj, "cx": float(c @ x), "step2": float(((x - xp) ** 2).sum())}


def _exact_diff(case, seed):
    lps = _models(case, seed)
    wx, wy = _adjoints(lps, seed)
    out = {k: [] for k in ("x", "y", "c", "a_val", "pobj")}
    n0 = m0 = 0
    for lp in lps:  # the unique vertex and its basis sensitivities
        x, y, f, d = lp.meta["x0"], lp.meta["y0"], lp.meta["interior"], lp.meta["tight"]
        dense = np.zeros((lp.m, lp.n))
        rows = np.repeat(np.arange(lp.m), np.diff(lp.A.ptr))
        dense[rows, lp.A.idx] = lp.A.val
        basis = dense[np.ix_(d, f)]
        p, q = np.zeros(lp.m), np.zeros(lp.n)
        p[d] = np.linalg.solve(basis.T, wx[n0:n0 + lp.n][f])
        q[f] = np.linalg.solve(basis, wy[m0:m0 + lp.m][d])
        n0, m0 = n0 + lp.n, m0 + lp.m
        for k, v in (("x", x), ("y", y), ("c", q), ("a_val", -(p[rows] * x[lp.A.idx] + y[rows] * q[lp.A.idx])),
                     ("pobj", [lp.c @ x])):
            out[k].append(v)
    return {**{k: np.concatenate(v) for k, v in out.items()}, "lo": None, "hi": None, "status": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "backend":
        return _exact_backend(case, seed)
    if kind == "diff":
        return _exact_diff(case, seed)
    return None
