"""Performance cases of the SPD factor-and-solve library: what a user has it do,
through its public entry points, from a single small system on host arrays to
the largest device-resident solve and thousands of small systems at once.

`listed()` names the cases, `draw(rng)` gives others of the same ranges,
`prepare` makes the inputs a caller would hold, `run` is one pass, `exact` the
same results from plain numpy or torch in 64 bits, and `work` the bytes and
operations that one pass cannot do without.

Host entry points (numpy views, the reference's trait methods) run with the
library's default algorithm choice; device entry points with the arguments that
a caller on a CUDA stream gives them.  Entry points that work in place get a
fresh copy of their input inside the pass, as a caller with new data brings one.
"""
import importlib
import math

import numpy as np
import torch

lla = importlib.import_module("linfa-linalg_gb300")


def listed():
    return [
        # one small covariance-sized system per call: launch and transfer latency
        {"name": "solvec_f64_n64", "kind": "solvec", "dtype": "f64", "n": 64, "m": 1, "order": "C"},
        # the single-matrix workload: n = 512, one right-hand side, row-major host arrays
        {"name": "solvec_f64_n512", "kind": "solvec", "dtype": "f64", "n": 512, "m": 1, "order": "C"},
        # a host solve above the reference-order limit (n > 1024), several right-hand sides
        {"name": "solvec_f64_n2048_r16", "kind": "solvec", "dtype": "f64", "n": 2048, "m": 16, "order": "C"},
        # the inverse of a covariance matrix (a precision matrix), column-major as ndarray's .t()
        {"name": "invc_f64_n300", "kind": "invc", "dtype": "f64", "n": 300, "m": 0, "order": "F"},
        # back substitution against an existing upper factor, single precision, ragged order
        {"name": "triangular_f32_n1000_r8", "kind": "triangular", "dtype": "f32", "n": 1000, "m": 8,
         "order": "C", "uplo": "upper"},
        # LOBPCG's Cholesky-QR of a tall block of vectors
        {"name": "orthonormalize_f64_n40000_k20", "kind": "orthonormalize", "dtype": "f64", "n": 40000, "m": 20,
         "order": "C"},
        # plain FP64 factor and solve of a matrix that already lies on the device (the
        # precision sweep's order and right-hand sides)
        {"name": "factor_solve_f64_n8192_r16", "kind": "factor_solve", "dtype": "f64", "n": 8192, "m": 16},
        # the same in single precision, ragged order, few right-hand sides
        {"name": "factor_solve_f32_n6001_r3", "kind": "factor_solve", "dtype": "f32", "n": 6001, "m": 3},
        # mixed-precision refined solve at the headline's size: n = 16384, 64 right-hand sides
        {"name": "refined_n16384_r64_slices", "kind": "refined", "n": 16384, "m": 64, "residual": "slices"},
        # a refined solve of ordinary size with the default options, ragged order
        {"name": "refined_n3001_r16_fp64", "kind": "refined", "n": 3001, "m": 16, "residual": "fp64"},
        # 10,000 uneven small systems (n 16..256, 1-8 right-hand sides) in one launch, both types
        {"name": "batch_f64_10000", "kind": "batch", "dtype": "f64", "count": 10000, "lo": 16, "hi": 256,
         "mode": "plain", "sizes": 1},
        {"name": "batch_f32_10000", "kind": "batch", "dtype": "f32", "count": 10000, "lo": 16, "hi": 256,
         "mode": "plain", "sizes": 1},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("solvec", "invc", "triangular", "orthonormalize", "factor_solve", "refined", "batch"))
    dtype, order = rng.choice(("f64", "f64", "f32")), rng.choice(("C", "F"))
    if kind == "solvec":
        return {"kind": kind, "dtype": dtype, "n": _log(rng, 16, 2048), "m": rng.randint(1, 16), "order": order}
    if kind == "invc":
        return {"kind": kind, "dtype": dtype, "n": _log(rng, 16, 1500), "m": 0, "order": order}
    if kind == "triangular":
        return {"kind": kind, "dtype": dtype, "n": _log(rng, 32, 2500), "m": rng.randint(1, 16), "order": order,
                "uplo": rng.choice(("upper", "lower"))}
    if kind == "orthonormalize":
        return {"kind": kind, "dtype": dtype, "n": _log(rng, 1000, 60000), "m": rng.randint(2, 48), "order": order}
    if kind == "factor_solve":
        return {"kind": kind, "dtype": dtype, "n": _log(rng, 256, 7000), "m": _log(rng, 1, 64)}
    if kind == "refined":
        return {"kind": kind, "n": _log(rng, 512, 9000), "m": _log(rng, 1, 64),
                "residual": rng.choice(("slices", "fp64"))}
    return {"kind": kind, "dtype": dtype, "count": _log(rng, 200, 8000), "lo": 16, "hi": _log(rng, 48, 256),
            "mode": "refined" if dtype == "f64" and rng.random() < 0.4 else "plain", "sizes": rng.randint(2, 999)}


# ---- inputs -----------------------------------------------------------------

def _np(case):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ordered(a, order):
    return np.asarray(a, order=order)


def _host_spd(n, dtype, seed):
    """A = G G^T / n + I, G i.i.d. N(0, 1), and the generator for what goes with it."""
    rng = np.random.default_rng(seed)
    g = rng.standard_normal((n, n))
    return (g @ g.T / n + np.eye(n)).astype(dtype), rng


def _device_spd(n, shift, g):
    """A = D (G G^T / n + shift I) D in FP64 on the device: features of unequal scale
    (D uniform in [1/2, 2)), full 53-bit entries; the product is formed in FP32."""
    G = torch.randn(n, n, device="cuda", generator=g)
    A = (G @ G.T).double().div_(n)
    del G
    A = (A + A.T).mul_(0.5)
    A.diagonal().add_(shift)
    d = torch.exp2(2 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g) - 1)
    return A.mul_(d[:, None]).mul_(d[None, :])


def _colmajor(t):
    """The same matrix with its columns contiguous."""
    return t.T.contiguous().T


def _batch_sizes(case):
    """Orders and right-hand sides of the systems: the caller's plan, the same for all inputs."""
    rng = np.random.default_rng(case["sizes"])
    n = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"] + 1), case["count"])).astype(np.int32)
    return np.clip(n, case["lo"], case["hi"]), rng.integers(1, 9, case["count"]).astype(np.int32)


def _batch_groups(plan):
    """Each order that occurs, with the indices of its systems."""
    for n in np.unique(plan.n):
        yield int(n), np.nonzero(plan.n == n)[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solvec", "invc"):
        a, rng = _host_spd(case["n"], _np(case), seed)
        a = _ordered(a, case["order"])
        s = {"case": case, "a": a, "work_a": np.empty_like(a)}
        if kind == "solvec":
            s["b"] = _ordered(rng.standard_normal((case["n"], case["m"])).astype(_np(case)), case["order"])
        return s
    if kind == "triangular":
        a, rng = _host_spd(case["n"], np.float64, seed)
        t = np.linalg.cholesky(a)
        t = (t if case["uplo"] == "lower" else t.T).astype(_np(case))
        b = rng.standard_normal((case["n"], case["m"])).astype(_np(case))
        return {"case": case, "t": _ordered(t, case["order"]), "b": _ordered(b, case["order"])}
    if kind == "orthonormalize":
        v = np.random.default_rng(seed).standard_normal((case["n"], case["m"])).astype(_np(case))
        return {"case": case, "v": _ordered(v, case["order"])}
    if kind == "factor_solve":
        g, n, dt = _gen(seed), case["n"], torch.float64 if case["dtype"] == "f64" else torch.float32
        A = _device_spd(n, 1.0, g).to(dt)
        A = torch.tril(A) + torch.tril(A, -1).T  # symmetric after the rounding to `dt` too
        B = _colmajor(torch.randn(n, case["m"], dtype=dt, device="cuda", generator=g))
        return {"case": case, "A": A.T, "B": B, "L": torch.empty_like(A).T, "X": _colmajor(torch.empty_like(B)),
                "info": torch.empty(1, dtype=torch.int64, device="cuda")}
    if kind == "refined":
        g, n = _gen(seed), case["n"]
        A = _device_spd(n, 0.1, g)  # a ridge-regularised Gram matrix
        A = torch.tril(A) + torch.tril(A, -1).T
        B = _colmajor(torch.randn(n, case["m"], dtype=torch.float64, device="cuda", generator=g))
        return {"case": case, "A": A.T, "B": B, "X": _colmajor(torch.empty_like(B))}
    if kind == "batch":
        n, m = _batch_sizes(case)
        plan = lla.BatchPlan(n, m, case["dtype"])
        dt = torch.float64 if case["dtype"] == "f64" else torch.float32
        g = _gen(seed)
        A = torch.zeros(plan.a_elems, dtype=dt, device="cuda")
        for k, at in _batch_groups(plan):
            G = torch.randn(len(at), k, k, device="cuda", generator=g)
            S = torch.bmm(G, G.mT).double().div_(k)
            S = (S + S.mT).mul_(0.5)
            S.diagonal(dim1=1, dim2=2).add_(0.1)
            off = torch.from_numpy(plan.a_off[at]).cuda()
            A[(off[:, None] + torch.arange(k * k, device="cuda")).reshape(-1)] = S.reshape(-1).to(dt)
        B = torch.randn(plan.b_elems, dtype=dt, device="cuda", generator=g)
        if case["mode"] == "refined":
            plan.set_refined()
        return {"case": case, "plan": plan, "A": A, "B": B, "work_a": torch.empty_like(A), "X": torch.empty_like(B),
                "info": torch.empty(case["count"], dtype=torch.int32, device="cuda")}
    raise ValueError(kind)


# ---- one pass ---------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solvec":
        np.copyto(s["work_a"], s["a"])  # solvec_inplace leaves the factor in its first argument
        return {"factor": s["work_a"], "x": lla.solvec(s["work_a"], s["b"])}
    if kind == "invc":
        np.copyto(s["work_a"], s["a"])
        return {"factor": s["work_a"], "inverse": lla.invc_inplace(s["work_a"])}
    if kind == "triangular":
        return lla.solve_triangular(s["t"], s["b"], case["uplo"])
    if kind == "orthonormalize":
        u, l = lla.orthonormalize(s["v"])
        return {"u": u, "l": l}
    st = torch.cuda.current_stream()
    if kind == "factor_solve":
        s["L"].copy_(s["A"])
        lla.potrf_device(s["L"], algo=lla.ALGO_FAST, info=s["info"], stream=st)
        s["X"].copy_(s["B"])
        lla.trsm_device(s["L"], s["X"], 0, algo=lla.ALGO_FAST, stream=st)
        lla.trsm_device(s["L"], s["X"], 1, algo=lla.ALGO_FAST, stream=st)
        return {"factor": s["L"], "x": s["X"], "info": s["info"]}
    if kind == "refined":
        lla.posv_refined_device(s["A"], s["B"], s["X"], stream=st, residual=case["residual"])
        return s["X"]
    s["X"].copy_(s["B"])
    if case["mode"] == "refined":
        s["plan"].solve_graph(s["A"], s["X"], s["info"], stream=st)
        return {"x": s["X"], "info": s["info"]}
    s["work_a"].copy_(s["A"])
    s["plan"].solve_graph(s["work_a"], s["X"], s["info"], stream=st)
    return {"factor": s["work_a"], "x": s["X"], "info": s["info"]}


# ---- the same in 64 bits ----------------------------------------------------

def _dirty(a, low):
    """The lower factor in the lower triangle, the rest as it was."""
    return np.tril(low) + np.triu(a.astype(np.float64), 1)


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("solvec", "invc"):
        a = s["a"].astype(np.float64)
        sym = np.tril(a) + np.tril(a, -1).T
        out = {"factor": _ordered(_dirty(s["a"], np.linalg.cholesky(sym)), case["order"])}
        if kind == "solvec":
            out["x"] = _ordered(np.linalg.solve(sym, s["b"].astype(np.float64)), case["order"])
        else:
            out["inverse"] = np.linalg.inv(sym)
        return out
    if kind == "triangular":
        return _ordered(np.linalg.solve(s["t"].astype(np.float64), s["b"].astype(np.float64)), case["order"])
    if kind == "orthonormalize":
        v = s["v"].astype(np.float64)
        low = np.linalg.cholesky(v.T @ v)
        return {"u": np.linalg.solve(low, v.T).T, "l": low}
    if kind == "factor_solve":
        A = s["A"].double()
        low = torch.linalg.cholesky(A)
        x = torch.cholesky_solve(s["B"].double(), low)
        return {"factor": torch.tril(low) + torch.triu(A, 1), "x": x, "info": None}
    if kind == "refined":
        return torch.cholesky_solve(s["B"], torch.linalg.cholesky(s["A"]))
    plan = s["plan"]
    factor, x = s["A"].double(), s["B"].double()
    for k, at in _batch_groups(plan):
        off = torch.from_numpy(plan.a_off[at]).cuda()
        ia = off[:, None] + torch.arange(k * k, device="cuda")
        S = factor[ia].reshape(len(at), k, k)
        low = torch.linalg.cholesky(S)
        # column-major in the pool: element (i, j) at i + j * k
        factor[ia.reshape(-1)] = (torch.tril(low) + torch.triu(S, 1)).mT.reshape(-1)
        for cols in range(1, 9):
            sel = np.nonzero(plan.m[at] == cols)[0]
            if not len(sel):
                continue
            ob = torch.from_numpy(plan.b_off[at[sel]]).cuda()
            ib = ob[:, None] + torch.arange(k * cols, device="cuda")
            rhs = x[ib].reshape(len(sel), cols, k).mT
            sol = torch.cholesky_solve(rhs, low[torch.from_numpy(sel).cuda()])
            x[ib.reshape(-1)] = sol.mT.reshape(-1)
    if case["mode"] == "refined":
        return {"x": x, "info": None}
    return {"factor": factor, "x": x, "info": None}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        n, m = (v.astype(np.float64) for v in _batch_sizes(case))
        esz, low = 8 if case["dtype"] == "f64" else 4, (n * (n + 1) / 2).sum()
        return {"bytes": float(esz * (low * (1 if case["mode"] == "refined" else 2) + 2 * (n * m).sum())),
                "flops": float((n ** 3 / 3 + 2 * n * n * m).sum())}
    n, m = float(case["n"]), float(case["m"])
    esz = 4 if case.get("dtype") == "f32" else 8
    low = n * (n + 1) / 2
    if kind in ("solvec", "factor_solve"):
        return {"bytes": esz * (2 * low + 2 * n * m), "flops": n ** 3 / 3 + 2 * n * n * m}
    if kind == "invc":
        return {"bytes": esz * (2 * low + n * n), "flops": n ** 3}
    if kind == "triangular":
        return {"bytes": esz * (low + 2 * n * m), "flops": n * n * m}
    if kind == "orthonormalize":
        return {"bytes": esz * (2 * n * m + m * m), "flops": 2 * n * m * m}
    return {"bytes": 8 * (low + 2 * n * m), "flops": n ** 3 / 3 + 2 * n * n * m}
