"""Performance cases of the PDHG engine: the calls a user of this library makes, over the
sizes it is used at, each through a public entry point with host arrays in and out (the
library's own interface) or, for the sparse primitives, with device vectors.

listed() are the cases that are followed by name, draw() gives others of the same ranges.
A case's "kind" is the entry point:

  spmv    A x and A'y with device vectors (the primitives a caller's own solver loops over)
  lp      fixed-step PDHG with scalar steps, lp_pdhg (an application that chose its steps)
  pre     fixed-step PDHG with per-row / per-column steps and the dual returned
  qp      fixed-step PDHG of a convex QP, general sparse or diagonal Hessian
  sk      sankhya_b200_pdhg_loop, the loop sk_solve hands a CSC model to
  pdlp    the restarted solve, FP64 or FP32 / bf16-valued iterations refined in FP64
  batch   many LPs of uneven size as one block-diagonal batch
  nodes   branch-and-bound node relaxations that share one matrix
  predict, gradient   the warm-start network, inference and one training gradient

Matrices follow the recipes of the-solver_b200/instances.py (uniform rows per column with
N(0,1) values; power-law columns with log-uniform magnitudes; the nonnegative packing matrix
of the node relaxations), generated on the GPU. Iteration counts are fixed and the
tolerances out of reach, so that a pass is the same work every time.
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_DEV = "cuda"
_F64 = torch.float64


def _engine():
    if "sankhya_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "sankhya_b200", os.path.join(_ROOT, "the-solver_b200", "__init__.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["sankhya_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["sankhya_b200"]


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one product and one transpose product of a small LP's matrix: a caller's own loop
        # pays the launch latency on every one
        {"name": "spmv_small", "kind": "spmv", "m": 2000, "n": 5000, "per_col": 5, "matrix": "uniform"},
        # the same on a ragged mid-size matrix
        {"name": "spmv_mid", "kind": "spmv", "m": 50021, "n": 100003, "per_col": 10, "matrix": "uniform"},
        # a small LP run with the caller's scalar steps, residuals every 100 iterations: the
        # reference's plain entry point at its small benchmark's size
        {"name": "lp_small", "kind": "lp", "m": 2000, "n": 5000, "per_col": 5, "matrix": "uniform",
         "iterations": 1000, "check_every": 100},
        # the headline workload: a power-law LP of 20M nonzeros, 100 iterations a call
        {"name": "lp_large", "kind": "pre", "m": 1000000, "n": 2000000, "per_col": 10, "matrix": "powerlaw",
         "iterations": 100, "check_every": 100},
        # a convex QP with an explicit sparse Hessian
        {"name": "qp_sparse", "kind": "qp", "m": 100000, "n": 200000, "per_col": 10, "matrix": "uniform",
         "hessian": "sparse", "iterations": 400, "check_every": 100},
        # the node LP or first-order LP of the C core's own solver, through its loop hook
        {"name": "sk_small", "kind": "sk", "m": 2000, "n": 5000, "per_col": 5, "matrix": "uniform",
         "iterations": 1000},
        # a small LP through the restarted solve (the default way to solve one)
        {"name": "pdlp_small", "kind": "pdlp", "m": 2000, "n": 5000, "per_col": 5, "matrix": "uniform",
         "precision": "fp64", "algorithm": "adaptive", "iterations": 2048},
        # a mid-size LP of the parametric family, mixed precision
        {"name": "pdlp_mid_fp32", "kind": "pdlp", "m": 50000, "n": 100000, "per_col": 10, "matrix": "uniform",
         "precision": "fp32", "algorithm": "adaptive", "iterations": 1024},
        # a large power-law LP, FP64, the Halpern iteration (the faster one on most instances)
        {"name": "pdlp_large", "kind": "pdlp", "m": 200000, "n": 400000, "per_col": 10, "matrix": "powerlaw",
         "precision": "fp64", "algorithm": "halpern", "iterations": 512},
        # many LPs of uneven size in one call
        {"name": "batch_uneven", "kind": "batch", "count": 512, "m_lo": 50, "m_hi": 5000, "iterations": 200},
        # node relaxations of one binary MILP, column bounds per node
        {"name": "nodes_256", "kind": "nodes", "m": 5000, "n": 10000, "per_col": 6, "batch": 256,
         "iterations": 1000},
        # one training gradient of the warm-start network (its forward pass is inference)
        {"name": "gradient", "kind": "gradient", "m": 50000, "n": 100000, "per_col": 10},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["spmv", "lp", "pre", "qp", "sk", "pdlp", "pdlp", "batch", "nodes", "predict", "gradient"])
    if kind == "batch":
        return {"kind": kind, "count": logint(12, 512), "m_lo": rng.randint(20, 60), "m_hi": logint(100, 5000),
                "iterations": rng.choice([60, 130, 200])}
    if kind == "nodes":
        m = logint(300, 5000)
        return {"kind": kind, "m": m, "n": 2 * m + rng.randint(0, 9), "per_col": rng.randint(3, 8),
                "batch": logint(5, 256), "iterations": rng.choice([100, 230, 500])}
    per_col = rng.randint(3, 12)
    if kind in ("predict", "gradient"):
        m = logint(300, 50000)
        return {"kind": kind, "m": m, "n": int(m * rng.uniform(1.5, 2.5)) + 1, "per_col": min(per_col, 10)}
    matrix = rng.choice(["uniform", "uniform", "powerlaw"])
    m = logint(200, {"qp": 100000, "sk": 20000, "pdlp": 150000}.get(kind, 300000))
    case = {"kind": kind, "m": m, "n": int(m * rng.uniform(1.2, 3.0)) + 1, "per_col": per_col, "matrix": matrix}
    if kind == "spmv":
        return case
    case["iterations"] = max(64, min(rng.choice([300, 512, 1000]), int(2e9 / (case["n"] * per_col))))
    if kind in ("lp", "pre", "qp"):
        case["check_every"] = rng.choice([20, 50, 100])
    if kind == "qp":
        case["hessian"] = rng.choice(["sparse", "diagonal"])
    if kind == "pdlp":
        case["precision"] = rng.choice(["fp64", "fp64", "fp32", "bf16"])
        case["algorithm"] = rng.choice(["adaptive", "adaptive", "halpern"]) if case["precision"] == "fp64" else "adaptive"
        if case["precision"] == "fp64" and case["algorithm"] == "adaptive":
            # the adaptive step amplifies the last bit: past this many iterations two FP64
            # evaluations of the same solve (this library's and exact()'s) are no longer near
            # each other (uniform 5e-12 after 128, power-law 9e-12 after 64, then 1e-7 and up)
            case["iterations"] = 128 if matrix == "uniform" else 64
    return case


# ------------------------------------------------------- instances (torch, GPU)

def _gen(seed):
    g = torch.Generator(device=_DEV)
    g.manual_seed(seed)
    return g


def _uniform(g, size, lo=0.0, hi=1.0):
    return torch.rand(size, generator=g, device=_DEV, dtype=_F64) * (hi - lo) + lo


def _normal(g, size):
    return torch.randn(size, generator=g, device=_DEV, dtype=_F64)


def _row_sums(ptr, v):
    """Sum of each row's consecutive values, in one fixed order."""
    return torch.segment_reduce(v, "sum", offsets=ptr, initial=0.0)


def _pattern(m, n, row, col):
    """CSR pattern of the distinct (row, col) pairs: offsets, columns, rows."""
    key = torch.unique(row * n + col)
    row = torch.div(key, n, rounding_mode="floor")
    ptr = torch.zeros(m + 1, dtype=torch.int64, device=_DEV)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
    return ptr, key - row * n, row


def _matrix(g, case):
    """(ptr, col, row, val) of a case's matrix."""
    m, n, per_col = case["m"], case["n"], case["per_col"]
    if case.get("matrix") == "powerlaw":
        # column degrees Pareto(1/2), the tail of Zipf(1.5), capped at 1,000, scaled to per_col on average
        raw = torch.clamp(torch.floor(_uniform(g, n, 1e-9).pow(-2.0)), max=1000.0)
        deg = torch.clamp(torch.round(raw * (per_col * n / float(raw.sum()))), 1, min(1000, m)).to(torch.int64)
    else:
        deg = torch.full((n,), per_col, dtype=torch.int64, device=_DEV)
    col = torch.repeat_interleave(torch.arange(n, device=_DEV), deg)
    row = torch.randint(0, m, (col.shape[0],), generator=g, device=_DEV)
    ptr, col, row = _pattern(m, n, row, col)
    nnz = col.shape[0]
    if case.get("matrix") == "powerlaw":
        val = 10.0 ** _uniform(g, nnz, -3.0, 3.0)
        val = torch.where(_uniform(g, nnz) < 0.5, -val, val)
    elif case["kind"] == "nodes":
        val = _uniform(g, nnz, 1.0, 10.0)
    else:
        val = _normal(g, nnz)
    return ptr, col, row, val


def _instance(case, seed):
    """The model of a case as device tensors: CSR A, c, bounds (and Q, targets, nodes)."""
    g = _gen(seed)
    kind = case["kind"]
    d = {}
    if kind == "batch":
        # m log-uniform, n = 2m, 4 to 8 entries per column, block-diagonal
        # (the sizes belong to the case, their order in the batch to the seed)
        k = case["count"]
        ms = torch.exp(torch.linspace(math.log(case["m_lo"]), math.log(case["m_hi"]), k, dtype=_F64)).to(torch.int64)
        ms = ms.to(_DEV)[torch.argsort(torch.rand(k, generator=g, device=_DEV))]
        zero = torch.zeros(1, dtype=torch.int64, device=_DEV)
        rseg = torch.cat([zero, torch.cumsum(ms, 0)])
        cseg = 2 * rseg
        m, n = int(rseg[-1]), int(cseg[-1])
        lp = torch.repeat_interleave(torch.arange(case["count"], device=_DEV), 2 * ms)
        deg = torch.randint(4, 9, (n,), generator=g, device=_DEV)
        col = torch.repeat_interleave(torch.arange(n, device=_DEV), deg)
        u = _uniform(g, col.shape[0])
        own = lp[col]
        row = rseg[own] + torch.minimum((u * ms[own]).to(torch.int64), ms[own] - 1)
        ptr, col, row = _pattern(m, n, row, col)
        val = _normal(g, col.shape[0])
        d.update(rseg=rseg, cseg=cseg)
    else:
        m, n = case["m"], case["n"]
        ptr, col, row, val = _matrix(g, case)
    d.update(m=m, n=n, ptr=ptr, col=col, row=row, val=val)
    if kind == "nodes":
        full = lambda k, v: torch.full((k,), v, dtype=_F64, device=_DEV)
        d.update(c=-_uniform(g, n), rl=full(m, -1e30), ru=0.3 * _row_sums(ptr, val))
        cl = torch.zeros((case["batch"], n), dtype=_F64, device=_DEV)
        cu = torch.ones((case["batch"], n), dtype=_F64, device=_DEV)
        # 1 to 50 variables of every node fixed to 0 or 1
        which = torch.randint(0, n, (case["batch"], 50), generator=g, device=_DEV)
        count = torch.randint(1, 51, (case["batch"], 1), generator=g, device=_DEV)
        live = torch.arange(50, device=_DEV)[None, :] < count
        node = torch.arange(case["batch"], device=_DEV)[:, None].expand(-1, 50)
        at = torch.unique((node * n + which)[live])
        to = torch.randint(0, 2, (at.shape[0],), generator=g, device=_DEV).to(_F64)
        cl.view(-1)[at] = to
        cu.view(-1)[at] = to
        d.update(cl=cl, cu=cu)
        return d
    lo, hi = (-5.0, 5.0) if kind == "qp" else (0.0, 10.0)
    x0 = _uniform(g, n, lo, hi)
    act = _row_sums(ptr, val * x0[col])
    d.update(c=_normal(g, n), rl=act - _uniform(g, m), ru=act + _uniform(g, m),
             cl=torch.full((n,), lo, dtype=_F64, device=_DEV), cu=torch.full((n,), hi, dtype=_F64, device=_DEV))
    if kind == "spmv":
        d.update(x=x0, y=_normal(g, m))
    if kind in ("lp", "pre", "qp"):
        a = val.abs()
        row_mass = _row_sums(ptr, a)
        order = torch.argsort(col, stable=True)
        cptr = torch.zeros(n + 1, dtype=torch.int64, device=_DEV)
        cptr[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
        col_mass = _row_sums(cptr, a[order])
        if kind == "lp":
            step = 0.9 / math.sqrt(float(row_mass.max()) * float(col_mass.max()))
            d.update(tau=step, sigma=step)
    if kind == "qp":
        diag = 10.0 ** _uniform(g, n, -2.0, 2.0)
        if case["hessian"] == "sparse":
            # Q = diag + L L', L with 3 entries N(0, 0.1) per column
            lr = torch.randint(0, n, (n, 3), generator=g, device=_DEV)
            lv = 0.1 * _normal(g, 3 * n).view(n, 3)
            key = torch.cat([(lr[:, :, None] * n + lr[:, None, :]).reshape(-1), torch.arange(n, device=_DEV) * (n + 1)])
            v = torch.cat([(lv[:, :, None] * lv[:, None, :]).reshape(-1), diag])
            order = torch.argsort(key, stable=True)
            key, counts = torch.unique_consecutive(key[order], return_counts=True)
            at = torch.zeros(key.shape[0] + 1, dtype=torch.int64, device=_DEV)
            at[1:] = torch.cumsum(counts, 0)
            qv = _row_sums(at, v[order])
            qr = torch.div(key, n, rounding_mode="floor")
            qptr = torch.zeros(n + 1, dtype=torch.int64, device=_DEV)
            qptr[1:] = torch.cumsum(torch.bincount(qr, minlength=n), 0)
            d.update(q_ptr=qptr, q_col=key - qr * n, q_row=qr, q_val=qv)
            col_mass = col_mass + _row_sums(qptr, qv.abs())
        else:
            d.update(qdiag=diag)
            col_mass = col_mass + diag
    if kind in ("pre", "qp"):
        d.update(tau=0.9 / (1.0 + col_mass), sigma=0.9 / (1.0 + row_mass))
    if kind in ("predict", "gradient"):
        r = np.random.RandomState(seed % (1 << 31))
        d["theta"] = np.concatenate([(r.uniform(-a, a, size=s)).astype(np.float32) for a, s in _theta_parts()])
        d.update(x_t=_uniform(g, n, lo, hi), y_t=_normal(g, m))
    return d


_ROUNDS, _H, _FEAT = 4, 64, 16


def _theta_parts():
    """(half width, length) of the network's parameters in the order of its flat vector."""
    parts = [(math.sqrt(6.0 / _FEAT), _FEAT * _H), (0.1, _H)] * 2
    parts += [(math.sqrt(6.0 / (2 * _H)), 2 * _H * _H), (0.1, _H)] * (2 * _ROUNDS)
    return parts + [(0.1, _H), (0.1, 1)] * 2


# ---------------------------------------------------------------- the calls

class _Csc(C.Structure):
    _fields_ = [("nrow", C.c_int), ("ncol", C.c_int), ("p", C.c_void_p), ("i", C.c_void_p), ("x", C.c_void_p),
                ("nzmax", C.c_int)]


class _Model(C.Structure):
    _fields_ = [("nrow", C.c_int), ("ncol", C.c_int), ("A", _Csc), ("Q", C.c_void_p)] + \
        [(k, C.c_void_p) for k in ("c", "rlow", "rupp", "clow", "cupp", "vartype")] + \
        [("objshift", C.c_double), ("objsense", C.c_double), ("rowname", C.c_void_p), ("colname", C.c_void_p),
         ("name", C.c_void_p)]


class _Options(C.Structure):
    _fields_ = [(k, C.c_double) for k in ("primal_tol", "dual_tol", "pivot_tol", "time_limit")] + \
        [("iteration_limit", C.c_longlong), ("node_limit", C.c_longlong)] + \
        [(k, C.c_int) for k in ("presolve", "scaling", "refactor_interval", "verbosity", "threads")] + \
        [("mip_gap_abs", C.c_double), ("mip_gap_rel", C.c_double)] + \
        [(k, C.c_int) for k in ("mip_cuts", "mip_heuristics", "dual_simplex", "lp_engine")] + \
        [("random_seed", C.c_ulonglong)]


def _pinned(t):
    """A page-locked host copy, as numpy."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    E = _engine()
    d = _instance(case, seed)
    kind, m, n = case["kind"], d["m"], d["n"]
    s = {"case": case, "kind": kind, "m": m, "n": n}
    if kind == "sk":
        order = torch.argsort(d["col"], stable=True)
        cptr = torch.zeros(n + 1, dtype=torch.int64, device=_DEV)
        cptr[1:] = torch.cumsum(torch.bincount(d["col"], minlength=n), 0)
        keep = {"p": _host(cptr.to(torch.int32)), "i": _host(d["row"][order].to(torch.int32)),
                "x": _host(d["val"][order])}
        keep.update({k: _host(d[k]) for k in ("c", "rl", "ru", "cl", "cu")})
        at = lambda k: keep[k].ctypes.data
        model = _Model(m, n, _Csc(m, n, at("p"), at("i"), at("x"), keep["x"].shape[0]), None, at("c"), at("rl"),
                       at("ru"), at("cl"), at("cu"), None, 0.0, 1.0, None, None, None)
        opts = _Options(primal_tol=1e-12, dual_tol=1e-12, iteration_limit=case["iterations"])
        s.update(keep=keep, model=model, opts=opts)
        return s
    s["A"] = E.Matrix(m, n, _host(d["ptr"].to(torch.int32)), _host(d["col"].to(torch.int32)), _host(d["val"]))
    if kind == "spmv":
        s.update(x=d["x"], y=d["y"], ax=torch.empty(m, dtype=_F64, device=_DEV),
                 aty=torch.empty(n, dtype=_F64, device=_DEV))
        return s
    s["inst"] = {k: _pinned(d[k]) for k in ("c", "rl", "ru", "cl", "cu")}
    if kind in ("lp", "pre", "qp"):
        scalar = kind == "lp"
        s["settings"] = E.settings(max_iterations=case["iterations"], check_every=case["check_every"],
                                   tau=d["tau"] if scalar else 1.0, sigma=d["sigma"] if scalar else 1.0,
                                   theta=1.0, tolerance=1e-14)
        s["x_out"] = _pinned(torch.zeros(n, dtype=_F64))
        s["y_out"] = None if scalar else _pinned(torch.zeros(m, dtype=_F64))
        if not scalar:
            s["tau"], s["sigma"] = _pinned(d["tau"]), _pinned(d["sigma"])
        if "qdiag" in d:
            s["qdiag"] = _pinned(d["qdiag"])
        if "q_val" in d:
            s["Q"] = E.Matrix(n, n, _host(d["q_ptr"].to(torch.int32)), _host(d["q_col"].to(torch.int32)),
                              _host(d["q_val"]))
    elif kind == "pdlp":
        p = E.pdlp_default_settings()
        p.max_iterations = case["iterations"]
        p.eps_optimal = 1e-13
        p.precision = {"fp64": E.FP64, "fp32": E.FP32_REFINE, "bf16": E.BF16_REFINE}[case["precision"]]
        p.algorithm = {"adaptive": E.PDLP_ADAPTIVE, "halpern": E.PDLP_HALPERN}[case["algorithm"]]
        s["settings"] = p
    elif kind in ("batch", "nodes"):
        b = E.batch_default_settings()
        b.max_iterations, b.check_every = case["iterations"], 20
        b.primal_tol = b.dual_tol = 1e-13
        s["settings"] = b
        if kind == "batch":
            s["rseg"], s["cseg"] = (_host(d[k].to(torch.int32)) for k in ("rseg", "cseg"))
    else:
        s["net"] = E.Gnn(rounds=_ROUNDS, seed=1, learning_rate=1e-3, y_scale=1.0)
        s["net"].set_parameters(d["theta"])
        s["x_t"], s["y_t"] = _pinned(d["x_t"]), _pinned(d["y_t"])
    return s


def _must(rc):
    if rc != 0:
        raise RuntimeError("the engine failed (%d): %s" % (rc, _engine().last_error()))


def run(s):
    E, kind, m, n = _engine(), s["kind"], s["m"], s["n"]
    if kind == "spmv":
        L, h = E.lib(), C.byref(s["A"].handle)
        _must(L.sankhya_cuda_spmv_device_f64(h, s["x"].data_ptr(), s["ax"].data_ptr()))
        _must(L.sankhya_cuda_spmv_transpose_device_f64(h, s["y"].data_ptr(), s["aty"].data_ptr()))
        return {"ax": s["ax"], "aty": s["aty"]}
    if kind in ("lp", "pre", "qp"):
        rc, x, y, r = E.pdhg(s["A"], s["inst"], s["settings"], hessian=s.get("Q"), qdiag=s.get("qdiag"),
                             primal_steps=s.get("tau"), dual_steps=s.get("sigma"), want_dual=kind != "lp",
                             x_out=s["x_out"], y_out=s["y_out"])
        _must(rc)
        return {"x": x, "y": y, "objective": r["objective"], "iterations": r["iterations"], "status": r["status"]}
    if kind == "sk":
        x, y, act = np.zeros(n), np.zeros(m), np.zeros(m)
        r = E.LoopResult()
        _must(E.lib().sankhya_b200_pdhg_loop(C.byref(s["model"]), C.byref(s["opts"]), E._p(x), E._p(y), E._p(act),
                                             C.byref(r)))
        return {"x": x, "y": y, "activity": act, "iterations": r.iterations}
    if kind == "pdlp":
        rc, x, y, r = E.pdlp_solve(s["A"], s["inst"], s["settings"])
        _must(rc)
        return {"x": x, "y": y, "iterations": r["iterations"], "status": r["status"]}
    if kind == "batch":
        rc, x, y, r = E.batch_pdhg(s["A"], s["inst"], s["rseg"], s["cseg"], s["settings"], want_dual=True)
        _must(rc)
        return {"x": x, "y": y, "objective": np.array([k["objective"] for k in r]),
                "iterations": np.array([k["iterations"] for k in r])}
    if kind == "nodes":
        i = s["inst"]
        rc, x, y, r = E.shared_batch_pdhg(s["A"], s["case"]["batch"], i["c"], i["rl"], i["ru"], i["cl"], i["cu"],
                                          s["settings"], want_dual=True)
        _must(rc)
        return {"x": x, "y": y, "objective": np.array([k["objective"] for k in r]),
                "iterations": np.array([k["iterations"] for k in r])}
    if kind == "predict":
        x, y = s["net"].predict(s["A"], s["inst"])
        return {"x": x, "y": y}
    loss, grad = s["net"].gradient(s["A"], s["inst"], s["x_t"], s["y_t"])
    return {"loss": loss, "gradient": grad}


# ------------------------------------------------------------ what it costs

def work(case):
    """Bytes and operations of a pass. One iteration depends on the one before it, so it
    reads the matrix in both orientations (12 bytes an entry, 4 an offset) and every vector
    its two steps need once, and writes their results once."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi = case["m_lo"], case["m_hi"]
        m = int(case["count"] * (hi - lo) / max(math.log(hi / lo), 1e-9))
        n, nnz = 2 * m, 12 * m
    else:
        m, n = case["m"], case["n"]
        nnz = case["n"] * case["per_col"]
    matrix = 2 * 12 * nnz + 4 * (m + n)
    if kind == "spmv":
        return {"bytes": matrix + 2 * 8 * (m + n), "flops": 4 * nnz}
    if kind in ("predict", "gradient"):
        # per round two dense layers (128 x 64 per node) and two aggregations of 64 channels
        nodes = m + n
        layer = nodes * 4 * (2 * _H) + 4 * 64 * nodes + matrix
        flops = _ROUNDS * (2 * 2 * _H * _H * nodes + 4 * _H * nnz) + 2 * _FEAT * _H * nodes
        k = 3 if kind == "gradient" else 1
        return {"bytes": k * _ROUNDS * layer, "flops": k * flops}
    width = case.get("batch", 1)
    vectors = width * (8 * n + 24 * m + 8 * m + 8 * m + 32 * n + 16 * n) if width == 1 else \
        8 * width * (2 * m + n + m + 5 * n) + 16 * (m + n)
    size = 8
    if kind == "pdlp":
        size = {"fp64": 8, "fp32": 4, "bf16": 4}[case["precision"]]
        value = {"fp64": 8, "fp32": 4, "bf16": 2}[case["precision"]]
        matrix = 2 * (4 + value) * nnz + 4 * (m + n)
        vectors = size * (10 * m + 8 * n)
    if kind == "qp" and case["hessian"] == "sparse":
        matrix += 12 * 10 * n + 4 * n
        vectors += 16 * n
    io = 8 * width * (3 * n + 2 * m) if kind != "nodes" else 8 * width * (3 * n + m)
    return {"bytes": case["iterations"] * (matrix + vectors) + io, "flops": case["iterations"] * 4 * nnz * width}


# ----------------------------------------------------- the same in 64 bits

def _sparse(ptr, col, val, rows, cols):
    return torch.sparse_csr_tensor(ptr, col, val, size=(rows, cols))


def _pair(d, val=None):
    """A and A' as torch sparse matrices."""
    val = d["val"] if val is None else val
    order = torch.argsort(d["col"], stable=True)
    cptr = torch.zeros(d["n"] + 1, dtype=torch.int64, device=_DEV)
    cptr[1:] = torch.cumsum(torch.bincount(d["col"], minlength=d["n"]), 0)
    return (_sparse(d["ptr"], d["col"], val, d["m"], d["n"]),
            _sparse(cptr, d["row"][order], val[order], d["n"], d["m"]))


def _clamp(v, lo, hi):
    return torch.minimum(torch.maximum(v, lo), hi)


def _plain_pdhg(d, iterations, tau, sigma, Q=None, qdiag=None):
    """x, y and A x_bar of the last dual step, of fixed-step PDHG from the box-clamped origin."""
    A, AT = _pair(d)
    wide = d["cl"].dim() == 2
    t = (lambda v: v.t().contiguous()) if wide else (lambda v: v)
    col = (lambda v: v[:, None]) if wide else (lambda v: v)
    c, rl, ru, cl, cu = col(d["c"]), col(d["rl"]), col(d["ru"]), t(d["cl"]), t(d["cu"])
    tau = col(tau) if torch.is_tensor(tau) else tau
    sigma = col(sigma) if torch.is_tensor(sigma) else sigma
    x = _clamp(torch.zeros_like(cl), cl, cu)
    x_bar = x.clone()
    y = torch.zeros((d["m"],) + tuple(x.shape[1:]), dtype=_F64, device=_DEV)
    for _ in range(iterations):
        v = y + sigma * (A @ x_bar)
        y = v - sigma * _clamp(v / sigma, rl, ru)
        g = c + AT @ y
        if Q is not None:
            g = g + Q @ x
        step = x - tau * g
        if qdiag is not None:
            step = step / (1.0 + tau * qdiag)
        new = _clamp(step, cl, cu)
        x_bar = 2.0 * new - x
        x = new
    return (x.t(), y.t()) if wide else (x, y)


def _scaled(d):
    """Ruiz to 1e-2, then Pock-Chambolle; the scaled model and its factors."""
    m, n, a = d["m"], d["n"], d["val"].abs()
    order = torch.argsort(d["col"], stable=True)
    cptr = torch.zeros(n + 1, dtype=torch.int64, device=_DEV)
    cptr[1:] = torch.cumsum(torch.bincount(d["col"], minlength=n), 0)
    red = lambda p, v, how: torch.segment_reduce(v, how, offsets=p, initial=0.0)
    R, S = torch.ones(m, dtype=_F64, device=_DEV), torch.ones(n, dtype=_F64, device=_DEV)
    done = False
    for _ in range(100):
        rn = R * red(d["ptr"], a * S[d["col"]], "max")
        cn = S * red(cptr, (a * R[d["row"]])[order], "max")
        dev = max(float(torch.where(v > 0, (v - 1).abs(), torch.zeros_like(v)).max()) for v in (rn, cn))
        if dev < 1e-2:
            done = True
            break
        R = torch.where(rn > 0, R / rn.clamp(min=1e-300).sqrt(), R)
        S = torch.where(cn > 0, S / cn.clamp(min=1e-300).sqrt(), S)
    if not done:
        R, S = torch.ones_like(R), torch.ones_like(S)
    v = a * R[d["row"]] * S[d["col"]]
    rs, cs = red(d["ptr"], v, "sum"), red(cptr, v[order], "sum")
    R = R * torch.where(rs > 0, rs.clamp(min=1e-300).rsqrt(), torch.ones_like(rs))
    S = S * torch.where(cs > 0, cs.clamp(min=1e-300).rsqrt(), torch.ones_like(cs))
    val = d["val"] * R[d["row"]] * S[d["col"]]
    return val, d["c"] * S, d["cl"] / S, d["cu"] / S, d["rl"] * R, d["ru"] * R, R, S


def _pdlp(d, case):
    """The restarted solve: adaptive steps, or reflected Halpern iterations."""
    val, c, cl, cu, rl, ru, R, S = _scaled(d)
    A, AT = _pair(d, val)
    dot = lambda u, v: float(torch.dot(u, v))
    cn, bn = math.sqrt(dot(c, c)), math.sqrt(dot(rl, rl) + dot(ru, ru))
    v = torch.full((d["n"],), 1.0 / math.sqrt(d["n"]), dtype=_F64, device=_DEV)
    sq = 1.0
    for _ in range(30):
        w = AT @ (A @ v)
        sq = dot(w, w)
        v = w / math.sqrt(sq)
    norm = math.sqrt(math.sqrt(sq))

    def worst(x, y, moves):
        ax, r = A @ x, c + AT @ y
        pr = ax - _clamp(ax, rl, ru)
        support = torch.where(y > 0, y * ru, y * rl)
        pobj = dot(c, x)
        dobj = float(torch.minimum(r * cl, r * cu).sum()) - float(support.sum())
        gap = abs(pobj - dobj) / (1.0 + abs(pobj) + abs(dobj))
        return max(math.sqrt(dot(pr, pr)) / (1.0 + bn), gap), ax, [math.sqrt(dot(u, u)) for u in moves]

    eta, omega = 0.9 / norm, min(1e6, max(1e-6, cn / bn))
    lo, hi = 1e-6 / norm, 1e4 / norm
    x, y = torch.zeros_like(c), torch.zeros_like(rl)
    xr, yr = x, y
    total, period, since, mu0, last, probes = case["iterations"], 64, 0, math.inf, math.inf, 0
    done = 0

    def reweigh(pm, dm, floor):
        if pm > floor and dm > floor:
            return min(1e6, max(1e-6, math.exp(0.5 * math.log(dm / pm) + 0.5 * math.log(omega))))
        return omega

    if case["algorithm"] == "halpern":
        while done < total:
            k = min(period, total - done)
            tau, sigma = eta / omega, eta * omega
            for q in range(k):
                lam = (since + q + 1.0) / (since + q + 2.0)
                xb = 2.0 * _clamp(x - tau * (c + AT @ y), cl, cu) - x
                x = lam * xb + (1.0 - lam) * xr
                v = y + sigma * (A @ xb)
                y = lam * (2.0 * (v - sigma * _clamp(v / sigma, rl, ru)) - y) + (1.0 - lam) * yr
            xt = _clamp(x - tau * (c + AT @ y), cl, cu)
            v = y + sigma * (A @ (2.0 * xt - x))
            yt = v - sigma * _clamp(v / sigma, rl, ru)
            done, since = done + k, since + k
            res = math.sqrt(omega * dot(xt - x, xt - x) + dot(yt - y, yt - y) / omega)
            again = res <= 0.2 * mu0 or (res <= 0.8 * mu0 and res > last) or since >= 0.36 * done
            last = res
            if again:
                omega = reweigh(math.sqrt(dot(xt - xr, xt - xr)), math.sqrt(dot(yt - yr, yt - yr)), 1e-14)
                x, y, xr, yr, since, mu0, last = xt, yt, xt, yt, 0, res, math.inf
        return x * S, y * R
    ax = axp = A @ x
    xs, ys, terms = torch.zeros_like(x), torch.zeros_like(y), 0
    while done < total:
        k = min(period, total - done)
        for _ in range(k):
            sigma, tau = eta * omega, eta / omega
            v = y + sigma * (2.0 * ax - axp)
            yc = v - sigma * _clamp(v / sigma, rl, ru)
            xc = _clamp(x - tau * (c + AT @ yc), cl, cu)
            axc = A @ xc
            dx, dy = xc - x, yc - y
            sums = torch.stack([torch.dot(dx, dx), torch.dot(dy, dy), torch.dot(dy, axc - ax)]).tolist()
            probes += 1
            half = 0.5 * (omega * sums[0] + sums[1] / omega)
            limit = half / abs(sums[2]) if abs(sums[2]) > 0.0 and half > 0.0 else hi
            ok = eta <= limit
            new = min((1.0 - (probes + 1.0) ** -0.3) * limit, (1.0 + (probes + 1.0) ** -0.6) * eta)
            eta = min(max(new if new > 0.0 and math.isfinite(new) else eta, lo), hi)
            if ok:
                x, y, axp, ax = xc, yc, ax, axc
                xs, ys, terms = xs + xc, ys + yc, terms + 1
        done, since = done + k, since + k
        cur = worst(x, y, (x - xr, y - yr))
        xa, ya = xs / max(terms, 1), ys / max(terms, 1)
        avg = worst(xa, ya, (xa - xr, ya - yr))
        best = avg if avg[0] < cur[0] else cur
        mu = best[0]
        again = mu <= 0.2 * mu0 or (mu <= 0.8 * mu0 and mu > last) or since >= 0.36 * done
        last = mu
        if again:
            if best is avg:
                x, y, ax = xa, ya, avg[1]
            axp = ax
            omega = reweigh(best[2][0], best[2][1], 1e-14)
            xr, yr, xs, ys, terms = x, y, torch.zeros_like(x), torch.zeros_like(y), 0
            since, mu0, last = 0, mu, math.inf
    return x * S, y * R


def _network(d, targets):
    m, n = d["m"], d["n"]
    theta = torch.tensor(d["theta"], dtype=_F64, device=_DEV, requires_grad=targets)
    at = [0]

    def take(*shape):
        k = math.prod(shape)
        at[0] += k
        return theta[at[0] - k:at[0]].view(*shape)

    A, AT = _pair(d)
    a = d["val"].abs()
    mass = lambda M: torch.sparse_csr_tensor(M.crow_indices(), M.col_indices(), M.values().abs(), size=M.shape) @ \
        torch.ones(M.shape[1], dtype=_F64, device=_DEV)
    rnorm, cnorm = mass(A), mass(AT)
    rdeg, cdeg = (M.crow_indices().diff().to(_F64) for M in (A, AT))
    an, bs = max(float(rnorm.max()), float(cnorm.max())), max(float(d["cl"].abs().max()), float(d["cu"].abs().max()))
    rs = max(float(d["rl"].abs().max()), float(d["ru"].abs().max()))
    one, pad = torch.ones(1, dtype=_F64, device=_DEV), torch.zeros(1, dtype=_F64, device=_DEV)
    fv = torch.stack([d["c"] / d["c"].abs().max(), d["cl"] / bs, d["cu"] / bs, one.expand(n), one.expand(n),
                      cnorm / an, cdeg / max(float(cdeg.max()), 1.0), one.expand(n)] + [pad.expand(n)] * 8, 1)
    fc = torch.stack([d["rl"] / rs, d["ru"] / rs, one.expand(m), one.expand(m), rnorm / an,
                      rdeg / max(float(rdeg.max()), 1.0), one.expand(m)] + [pad.expand(m)] * 9, 1)
    del a
    ir, ic = 1.0 / rdeg.clamp(min=1.0)[:, None], 1.0 / cdeg.clamp(min=1.0)[:, None]

    class Product(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, M, MT):
            ctx.MT = MT
            return M @ x

        @staticmethod
        def backward(ctx, g):
            return ctx.MT @ g.contiguous(), None, None

    hv = torch.relu(fv @ take(_FEAT, _H) + take(_H))
    hc = torch.relu(fc @ take(_FEAT, _H) + take(_H))
    for _ in range(_ROUNDS):
        hc = torch.relu(torch.cat([hc, ir * Product.apply(hv, A, AT)], 1) @ take(2 * _H, _H) + take(_H))
        hv = torch.relu(torch.cat([hv, ic * Product.apply(hc, AT, A)], 1) @ take(2 * _H, _H) + take(_H))
    sx = hv @ take(_H) + take(1)
    y = hc @ take(_H) + take(1)
    width = d["cu"] - d["cl"]
    x = d["cl"] + width * torch.sigmoid(sx)
    if not targets:
        return {"x": _clamp(x, d["cl"], d["cu"]), "y": y}
    loss = (((x - d["x_t"]) / width) ** 2).mean() + ((y - d["y_t"]) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "gradient": theta.grad}


def exact(case, seed):
    d = _instance(case, seed)
    kind = case["kind"]
    if kind == "spmv":
        A, AT = _pair(d)
        return {"ax": A @ d["x"], "aty": AT @ d["y"]}
    if kind in ("predict", "gradient"):
        return _network(d, kind == "gradient")
    if kind == "pdlp":
        x, y = _pdlp(d, case)
        return {"x": x, "y": y, "iterations": None, "status": None}
    if kind in ("lp", "pre", "qp"):
        Q = _sparse(d["q_ptr"], d["q_col"], d["q_val"], d["n"], d["n"]) if "q_val" in d else None
        x, y = _plain_pdhg(d, case["iterations"], d["tau"], d["sigma"], Q, d.get("qdiag"))
        obj = torch.dot(d["c"], x)
        if Q is not None:
            obj = obj + 0.5 * torch.dot(x, Q @ x)
        if "qdiag" in d:
            obj = obj + 0.5 * torch.dot(x, d["qdiag"] * x)
        return {"x": x, "y": None if kind == "lp" else y, "objective": float(obj), "iterations": None,
                "status": None}
    # the diagonal steps of sk_solve
    A, AT = _pair(d)
    mass = lambda M: _sparse(M.crow_indices(), M.col_indices(), M.values().abs(), *M.shape) @ \
        torch.ones(M.shape[1], dtype=_F64, device=_DEV)
    x, y = _plain_pdhg(d, case["iterations"], 0.9 / (1.0 + mass(AT)), 0.9 / (1.0 + mass(A)))
    if kind == "sk":
        return {"x": x, "y": y, "activity": A @ x, "iterations": None}
    if kind == "nodes":
        return {"x": x, "y": y, "objective": x @ d["c"], "iterations": None}
    return {"x": x, "y": y, "iterations": None,
            "objective": torch.stack([torch.dot(d["c"][a:b], x[a:b]) for a, b in
                                      zip(d["cseg"][:-1].tolist(), d["cseg"][1:].tolist())])}
