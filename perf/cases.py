"""What a user has this package do, as a list of measurable cases.

``listed()`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes a
case's inputs from a seed, ``run`` is one pass through the public entry points, ``work``
says what the pass cannot do without and ``exact`` computes its energies in FP64 with plain
torch.

A case is one operation (``op``) on matrices of one kind:

* ``qbf``       QBF().solve(problem): the exhaustive search of one problem
* ``qbf1``      QB_F1().solve(problem): the int16 solver with its own tie order
* ``wrap``      the same with the reference's overflowing int16 arithmetic
* ``parallel``  Parallel(base_solver=QBF, splits_cnt=k) on one device
* ``minima``    QBF().solve with the energy_arr metric (every prefix's minimum)
* ``resident``  a Q that already lies in device memory, through the C ABI's binding
* ``batch``     thousands of small independent problems in one call
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qubo_b200  # noqa: F401  (makes the package importable under its import name)
from qubo_b200 import _lib
from qubo_b200.problems import Just_Q
from qubo_b200.solvers import QB_F1, QBF, Parallel

_DTYPES = {"f32": np.float32, "f64": np.float64, "i16": np.int16, "i32": np.int32}


def listed():
    return [
        # a tiny problem: the whole call is latency (inner loop of a heuristic, a unit test)
        {"name": "qbf_n14_f32", "op": "qbf", "kind": "uniform", "dtype": "f32", "n": 14},
        # RandomQUBO of 20 variables, symmetrised float entries in [-1, 1): still latency
        {"name": "qbf_n20_f32", "op": "qbf", "kind": "symmetric", "dtype": "f32", "n": 20},
        # an odd size whose double-precision matrix an earlier GPU step left in device memory
        {"name": "resident_n25_f64", "op": "resident", "kind": "normal", "dtype": "f64", "n": 25},
        # every prefix's minimum (the energy_arr metric: 2^7 prefixes of 2^20 states)
        {"name": "minima_n27_f32", "op": "minima", "kind": "uniform", "dtype": "f32", "n": 27},
        # 32-variable int16 matrix with entries in [-100, 100] for QB_F1
        {"name": "qbf1_n32_i16", "op": "qbf1", "kind": "symmetric", "dtype": "i16", "n": 32},
        # bit fixing into 8 tasks, as a user of the reference spreads a search over workers
        {"name": "parallel_n33_i32", "op": "parallel", "kind": "uniform", "dtype": "i32", "n": 33, "splits": 8},
        # the reference's int16 arithmetic, overflow included
        {"name": "wrap_n34_i16", "op": "wrap", "kind": "uniform", "dtype": "i16", "n": 34},
        # 6-city TSP with integer distances: 36 variables, the benchmark's workload
        {"name": "qbf_tsp6_i32", "op": "qbf", "kind": "tsp", "dtype": "i32", "n": 36},
        # the notebook's 37-variable random float matrix
        {"name": "qbf_n37_f32", "op": "qbf", "kind": "uniform", "dtype": "f32", "n": 37},
        # MaxCut on G(40, 0.5) with weights +-1: many ties, the longest single search here
        {"name": "qbf_maxcut40_i32", "op": "qbf", "kind": "maxcut", "dtype": "i32", "n": 40},
        # a few hundred small problems of mixed types, mostly below 20 variables
        {"name": "batch_300_mixed", "op": "batch", "kind": "mixed", "count": 300, "n_lo": 5, "n_hi": 22},
        # 4096 float problems with 16 to 28 variables in one call
        {"name": "batch_4096_f32", "op": "batch", "kind": "normal", "dtype": "f32", "count": 4096, "n_lo": 16,
         "n_hi": 28},
    ]


def draw(rng):
    op = rng.choice(["qbf", "qbf", "qbf", "qbf1", "parallel", "wrap", "minima", "resident", "batch", "batch"])
    if op == "batch":
        if rng.random() < 0.5:
            lo = rng.randint(4, 12)
            return {"op": op, "kind": "mixed", "count": int(math.exp(rng.uniform(math.log(20), math.log(600)))),
                    "n_lo": lo, "n_hi": rng.randint(lo + 4, 22)}
        lo = rng.randint(14, 22)
        return {"op": op, "kind": "normal", "dtype": rng.choice(["f32", "f64"]),
                "count": int(math.exp(rng.uniform(math.log(100), math.log(3000)))), "n_lo": lo,
                "n_hi": rng.randint(lo + 1, 27)}
    if op == "minima":
        return {"op": op, "kind": rng.choice(["uniform", "symmetric"]), "dtype": rng.choice(["f32", "f64", "i32"]),
                "n": rng.randint(21, 27)}
    if op in ("qbf1", "wrap"):
        return {"op": op, "kind": rng.choice(["uniform", "symmetric"]), "dtype": "i16",
                "n": rng.randint(21, 37 if op == "qbf1" else 35)}
    if op == "resident":
        return {"op": op, "kind": rng.choice(["normal", "symmetric"]), "dtype": rng.choice(["f32", "f64", "i32"]),
                "n": rng.randint(12, 35)}
    kind = rng.choice(["uniform", "symmetric", "normal", "maxcut", "tsp"])
    n = rng.randint(10, 38) if kind != "tsp" else rng.choice([16, 25, 36])
    dtype = "i32" if kind in ("maxcut", "tsp") else "f32" if kind == "normal" else \
        rng.choice(["f32", "f64", "i16", "i32"])
    case = {"op": op, "kind": kind, "dtype": dtype, "n": n}
    if op == "parallel":
        case["splits"] = rng.choice([2, 4, 8, 16])
    return case


# ------------------------------------------------------------------------------ inputs
def _matrix(kind: str, dtype: str, n: int, rng) -> np.ndarray:
    dt = _DTYPES[dtype]
    integer = np.issubdtype(dt, np.integer)
    if kind == "uniform":  # RandomQUBO's range: not symmetric
        return (rng.integers(-100, 100, (n, n)) if integer else rng.uniform(-100, 100, (n, n))).astype(dt)
    if kind == "symmetric":
        if integer:
            U = np.triu(rng.integers(-100, 101, (n, n)))
            return (U + np.triu(U, 1).T).astype(dt)
        U = rng.uniform(-1, 1, (n, n))
        return ((U + U.T) / 2).astype(dt)
    if kind == "normal":
        G = rng.standard_normal((n, n)) * (20 if integer else 1)
        G = (G + G.T) / 2
        return (np.rint(G) if integer else G).astype(dt)
    if kind == "maxcut":  # E(x) = -cut(x) of an Erdos-Renyi graph with weights +-1
        present = np.triu(rng.random((n, n)) < 0.5, 1)
        w = (rng.integers(0, 2, (n, n)) * 2 - 1) * present
        Q = 2 * w
        Q[np.arange(n), np.arange(n)] = -(w.sum(axis=0) + w.sum(axis=1))
        return Q.astype(dt)
    # tsp: integer distances, x[city * m + position], one-hot penalties of weight 2 max(w) + 1
    m = math.isqrt(n)
    w = np.triu(rng.integers(1, 101, (m, m)), 1)
    w = w + w.T
    city, pos = np.divmod(np.arange(n), m)
    nxt = pos[None, :] == pos[:, None] + 1
    Q = np.where(nxt, w[city[:, None], city[None, :]], 0)
    P = 2 * w.max() + 1
    same = (city[:, None] == city[None, :]) | (pos[:, None] == pos[None, :])
    Q = Q + P * np.where(np.eye(n, dtype=bool), -1, same)
    return (np.triu(Q) + np.tril(Q, -1).T).astype(dt)


def _matrices(case, seed):
    """The case's matrices: one, or the batch's list."""
    rng = np.random.default_rng([seed, 7])
    if case["op"] != "batch":
        return [_matrix(case["kind"], case["dtype"], case["n"], rng)]
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(case["n_lo"], case["n_hi"] + 1))
        if case["kind"] == "mixed":
            dtype = ("f32", "i16", "i32", "f64")[int(rng.integers(4))]
            out.append(_matrix("uniform" if dtype[0] == "i" else "normal", dtype, n, rng))
        else:
            out.append(_matrix(case["kind"], case["dtype"], n, rng))
    return out


def prepare(case, seed):
    Qs = _matrices(case, seed)
    op = case["op"]
    state = {"op": op}
    if op == "batch":
        state["Qs"] = Qs
        state["handle"] = _lib.handle(0)
    elif op == "resident":
        state["Q"] = torch.as_tensor(Qs[0], device="cuda")
        state["dtype"] = Qs[0].dtype
        state["handle"] = _lib.handle(0)
    else:
        state["problem"] = Just_Q(Qs[0])
        if op == "parallel":
            state["solver"] = Parallel(base_solver=QBF, splits_cnt=case["splits"], devices=["cuda"])
    return state


# --------------------------------------------------------------------------------- run
def run(state):
    op = state["op"]
    if op == "batch":
        r = state["handle"].solve_batch(state["Qs"], stream=torch.cuda.current_stream().cuda_stream)
        return {"best_E": r.best_E, "best_X": r.best_X_int.astype(np.int64)}
    if op == "resident":
        Q = state["Q"]
        r = state["handle"].solve_device(Q.data_ptr(), Q.shape[0], state["dtype"],
                                         stream=torch.cuda.current_stream().cuda_stream)
        return {"best_E": np.float64(r["best_E"]), "best_X": r["best_X"]}
    if op == "qbf":
        sol = QBF().solve(state["problem"], device="cuda")
    elif op == "qbf1":
        sol = QB_F1().solve(state["problem"], device="cuda")
    elif op == "wrap":
        sol = QB_F1().solve(state["problem"], device="cuda", int16_wrap=True)
    elif op == "parallel":
        sol = state["solver"].solve(state["problem"])
    else:
        sol = QBF().solve(state["problem"], device="cuda", use_metrics={"energy_arr"})
    out = {"best_E": sol.best_E, "best_X": sol.best_X}
    if op == "minima":
        out["energy_arr"] = sol.metrics[0]["energy_arr"]
    return out


# -------------------------------------------------------------------------------- work
def work(case):
    """Every state's energy from its neighbour's (one addition) and into the minimum (one
    comparison); the matrix in, the answer out."""
    if case["op"] == "batch":
        ns = range(case["n_lo"], case["n_hi"] + 1)
        per = case["count"] / len(ns)
        item = 5 if case["kind"] == "mixed" else np.dtype(_DTYPES[case["dtype"]]).itemsize
        return {"bytes": sum(per * (n * n * item + 16) for n in ns), "flops": sum(per * 2.0 * 2 ** n for n in ns)}
    n = case["n"]
    nbytes = n * n * np.dtype(_DTYPES[case["dtype"]]).itemsize + 8 + 4 * n
    if case["op"] == "minima":
        return {"bytes": nbytes + 8 * 2 ** max(0, n - 20), "flops": 4.0 * 2 ** n}  # the search and the metric
    return {"bytes": nbytes, "flops": 2.0 * 2 ** n}


# ------------------------------------------------------------------------------- exact
def _bits(values, width):
    """Rows of MSB-first bits (float64 on the GPU) of a tensor of integers."""
    shifts = torch.arange(width - 1, -1, -1, device=values.device)
    return ((values[:, None] >> shifts) & 1).to(torch.float64)


def _minima(Q: np.ndarray, keep: int):
    """min over x of x^T Q x for every value of the first ``keep`` variables (natural order),
    each energy evaluated once more from its state."""
    n = Q.shape[0]
    b = min(n - keep, 14)
    a = n - b
    Qd = torch.as_tensor(Q.astype(np.float64), device="cuda")
    S = _bits(torch.arange(1 << b, device="cuda"), b)
    C = Qd[:a, a:] + Qd[a:, :a].T
    St = torch.cat([S, ((S @ Qd[a:, a:]) * S).sum(1, keepdim=True)], dim=1).T.contiguous()
    best, arg = [], []
    for p0 in range(0, 1 << a, 1 << 14):
        P = _bits(torch.arange(p0, min(1 << a, p0 + (1 << 14)), device="cuda"), a)
        H = torch.cat([P @ C, P.new_ones(P.shape[0], 1)], dim=1)
        v, i = (H @ St).min(dim=1)
        if a:
            v = v + ((P @ Qd[:a, :a]) * P).sum(1)
        best.append(v)
        arg.append((torch.arange(p0, p0 + P.shape[0], device="cuda") << b) | i)
        if len(best) > 256:
            best, arg = _fold(best, arg, keep, a)
    best, arg = torch.cat(best), torch.cat(arg)
    v, i = best.reshape(1 << keep, -1).min(dim=1)
    x = _bits(arg.reshape(1 << keep, -1).gather(1, i[:, None])[:, 0], n)
    return ((x @ Qd) * x).sum(1).cpu().numpy()


def _fold(best, arg, keep, a):
    """Without kept variables only the smallest so far is needed (bounds the memory used)."""
    if keep:
        return best, arg
    v, x = torch.cat(best), torch.cat(arg)
    i = v.argmin()
    return [v[i:i + 1]], [x[i:i + 1]]


def exact(case, seed):
    Qs = _matrices(case, seed)
    op = case["op"]
    if op in ("wrap", "qbf1"):  # whole numbers throughout
        return None
    if op == "batch":
        return {"best_E": np.array([_minima(Q, 0)[0] for Q in Qs]), "best_X": None}
    out = {"best_E": _minima(Qs[0], 0)[0], "best_X": None}
    if op == "minima":
        A = case["n"] - 20
        i = np.arange(1 << A)
        out["energy_arr"] = _minima(Qs[0], A)[i ^ (i >> 1)]  # the prefixes in Gray order
    return out
