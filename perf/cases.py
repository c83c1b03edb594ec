"""Workloads of the solve phase, each through the entry point a program calls.

A program factors a graph and uploads it once, then solves many right-hand
sides with the handle, so `prepare` keeps one handle per graph (the last few)
and makes fresh right-hand sides from its seed.  Graphs and factors depend on
the case alone: the generators and the elimination are seeded.

Entries:
  call    f(b) on host arrays: DeviceLapSolver.__call__, the reference's closure
  device  acg_solve_device / acg_solve_batch_device on device memory
  apply   acg_ldlsolve_noalloc: one preconditioner application on device memory
  group   GroupSolver: many graphs, one right-hand side each, in one launch
  serve   ServeLoop: a burst of requests on the device-resident loop
"""
import ctypes
import math
import os
import random
import sys
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "laplacians.jl_b200"))

import acgpu  # noqa: E402
from acgpu import generators as G  # noqa: E402
from acgpu._lib import AcgSolveInfo, check, lib  # noqa: E402

_PREC = {"fp64": 0, "mixed": 1}
_MAXITS = 2000


def _case(name, entry, graph, dims, weights, rhs, precision, tol):
    return dict(name=name, entry=entry, graph=graph, dims=dims, weights=weights, rhs=rhs, precision=precision, tol=tol)


def listed():
    return [
        # the reference's default call (tol 1e-6, FP64) on a small graph: all latency
        _case("small_call", "call", "grid2", "32x32", "unit", 1, "fp64", 1e-6),
        # the 2D grid of the benchmark, one right-hand side, default tolerance
        _case("grid2_200_call", "call", "grid2", "200x200", "unit", 1, "fp64", 1e-6),
        # the 3D grid of the reference's documentation, weighted, device memory
        _case("grid3_50_device", "device", "grid3", "50x50x50", "loguniform", 1, "fp64", 1e-8),
        # a geometric graph (ragged degrees, weights 1/distance), mixed precision
        _case("geometric_call", "call", "geometric", "60000", "inverse_distance", 1, "mixed", 1e-10),
        # a path with four matchings: a deep factor with long columns
        _case("matchings_device", "device", "matchings", "150000", "lognormal:2", 1, "fp64", 1e-8),
        # the 1M-vertex grid, one right-hand side: latency of the largest graph
        _case("grid3_100_device", "device", "grid3", "100x100x100", "loguniform", 1, "mixed", 1e-10),
        # the benchmark's batch: 64 right-hand sides of the 1M-vertex grid
        _case("grid3_100_batch64", "device", "grid3", "100x100x100", "loguniform", 64, "mixed", 1e-10),
        # an odd grid and an odd number of right-hand sides in FP64 (padded columns)
        _case("grid3_odd_batch13", "device", "grid3", "61x53x47", "loguniform", 13, "fp64", 1e-8),
        # a few right-hand sides at once from host arrays
        _case("matchings_call5", "call", "matchings", "20000", "lognormal:2", 5, "mixed", 1e-10),
        # the preconditioner alone, as an outer solver of the caller's would apply it
        _case("apply_grid3_50", "apply", "grid3", "50x50x50", "loguniform", 1, "fp64", 0.0),
        # the components of a disconnected graph: 2D grids and geometric graphs
        _case("group_24", "group", "mix", "24x120", "mixed", 1, "fp64", 1e-8),
        # a burst of requests of 1 to 8 right-hand sides on the serving loop
        _case("serve_burst", "serve", "grid3", "30x30x30", "lognormal:1", 24, "mixed", 1e-10),
    ]


def draw(rng):
    """One more case of the same ranges: graphs of 700 to 1,000,000 vertices
    (the eliminations with long columns to 60,000), 1 to 64 right-hand sides."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["call", "call", "device", "device", "device", "apply", "group", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    tol = rng.choice([1e-6, 1e-8]) if precision == "fp64" else 1e-10
    if entry == "group":
        return _case("", "group", "mix", f"{logint(3, 24)}x{logint(40, 120)}", "mixed", 1, "fp64", tol if precision == "fp64" else 1e-8)
    rhs = 1 if rng.random() < 0.5 else logint(2, 64)
    top = 131072 if entry == "apply" else 1000000
    if entry == "serve":
        precision, tol, rhs, top = "mixed", 1e-10, logint(2, 24), 60000
    if entry == "apply":
        precision, tol, rhs = "fp64", 0.0, 1
    n = logint(700, top)
    graph = rng.choice(["grid2", "grid3", "geometric", "matchings"])
    if graph == "grid2":
        a = max(8, int(n ** 0.5 * rng.uniform(0.6, 1.6)))
        dims, weights = f"{a}x{max(8, n // a)}", rng.choice(["unit", "loguniform"])
    elif graph == "grid3":
        a = max(4, int(n ** (1 / 3) * rng.uniform(0.7, 1.4)))
        b = max(4, int((n / a) ** 0.5 * rng.uniform(0.8, 1.2)))
        dims, weights = f"{a}x{b}x{max(4, n // (a * b))}", rng.choice(["unit", "loguniform", "lognormal:1"])
    elif graph == "geometric":
        dims, weights = str(max(1000, min(n, 100000))), "inverse_distance"
    else:
        dims, weights = str(min(n, 60000)), "lognormal:2"
    c = _case("", entry, graph, dims, weights, rhs, precision, tol)
    del c["name"]
    return c


# ---- graphs and handles -------------------------------------------------------

def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _key(case):
    return case["graph"], case["dims"], case["weights"]


@lru_cache(maxsize=3)
def _graph(graph, dims, weights):
    d = tuple(int(v) for v in dims.split("x"))
    if graph == "grid2":
        return [G.grid2(*d, weights=weights, seed=1)]
    if graph == "grid3":
        return [G.grid3(*d, weights=weights, seed=1)]
    if graph == "geometric":
        return [G.largest_component(G.random_geometric(d[0], seed=1, weights=weights))]
    if graph == "matchings":
        return [G.path_plus_matchings(d[0], k=4, sigma=float(weights.split(":")[1]), seed=1)]
    # a group: half 2D grids, half geometric graphs, of mixed sizes
    count, side = d
    rng = random.Random(count * 1000 + side)
    out = []
    for i in range(count):
        if i % 2 == 0:
            out.append(G.grid2(rng.randint(32, side), rng.randint(32, side), weights="loguniform", seed=i))
        else:
            out.append(G.largest_component(G.random_geometric(rng.randint(1000, side * side), seed=i)))
    return out


@lru_cache(maxsize=3)
def _handle(entry, graph, dims, weights):
    graphs = _graph(graph, dims, weights)
    acgpu.seed(1)
    factors = [acgpu.approx_chol(a) for a in graphs]
    if entry == "group":
        return acgpu.GroupSolver(graphs, factors)
    solver = acgpu.DeviceLapSolver(graphs[0], factors[0])
    if entry == "serve":
        return acgpu.ServeLoop(solver, precision="mixed", slots=64, queue=64)
    return solver


def _requests(case):
    rng = random.Random(case["rhs"])
    return [rng.randint(1, 8) for _ in range(case["rhs"])]


def _columns(case):
    return sum(_requests(case)) if case["entry"] == "serve" else case["rhs"]


def _sizes(case):
    return [a.shape[0] for a in _graph(*_key(case))]


def _rhs(case, seed):
    """Gaussian right-hand sides without their mean (per graph), one row each."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    sizes = _sizes(case)
    b = torch.randn((_columns(case), sum(sizes)), generator=gen, device="cuda", dtype=torch.float64)
    at = 0
    for n in sizes:
        b[:, at:at + n] -= b[:, at:at + n].mean(dim=1, keepdim=True)
        at += n
    return b


def prepare(case, seed):
    kind = case["entry"] if case["entry"] in ("group", "serve") else "solve"
    state = {"case": case, "h": _handle(kind, *_key(case))}
    b = _rhs(case, seed)
    if case["entry"] == "device":
        state.update(b=b, x=torch.empty_like(b), info=(AcgSolveInfo * case["rhs"])())
    elif case["entry"] == "apply":
        state.update(b=b[0].contiguous(), x=torch.empty_like(b[0]))
    elif case["entry"] == "serve":
        cols, at, reqs = b.cpu().numpy().T, 0, []
        for k in _requests(case):
            reqs.append(np.ascontiguousarray(cols[:, at:at + k]))
            at += k
        state["b"] = reqs
    elif case["entry"] == "group":
        host, at, parts = b[0].cpu().numpy(), 0, []
        for n in _sizes(case):
            parts.append(host[at:at + n].copy())
            at += n
        state["b"] = parts
    else:
        host = b.cpu().numpy()
        state["b"] = host[0].copy() if case["rhs"] == 1 else np.ascontiguousarray(host.T)
    return state


def run(state):
    case, h, b = state["case"], state["h"], state["b"]
    tol, prec = case["tol"], _PREC[case["precision"]]
    # L x = b fixes x up to a constant per graph, and the FP32 inner solves leave
    # one in x: a program that wants the potentials themselves removes the mean
    mixed = case["precision"] == "mixed"
    if case["entry"] == "call":
        x = h(b, tol=tol, maxits=_MAXITS, precision=case["precision"])
        return x - x.mean(axis=0) if mixed else x
    if case["entry"] == "group":
        xs = h(b, tol=tol, maxits=_MAXITS, precision=case["precision"])
        return xs
    if case["entry"] == "serve":
        tickets = [h.submit(r, tol=tol, maxits=_MAXITS) for r in b]
        xs = [t.wait() for t in tickets]
        return [x - x.mean(axis=0) for x in xs]
    x = state["x"]
    if case["entry"] == "apply":
        check(lib().acg_ldlsolve_noalloc(h._h, b.data_ptr(), x.data_ptr(), prec, None))
    elif case["rhs"] == 1:
        check(lib().acg_solve_device(h._h, b.data_ptr(), x.data_ptr(), tol, _MAXITS, math.inf, 5, prec, state["info"]))
    else:
        check(lib().acg_solve_batch_device(h._h, b.data_ptr(), x.data_ptr(), case["rhs"], h.n, tol, _MAXITS, math.inf,
                                           5, prec, state["info"]))
    return x.sub_(x.mean(dim=1, keepdim=True)) if mixed else x


# Entries per vertex of the adjacency and of the factor, by family (the
# eliminations of these generators), and about 3.75 PCG iterations a digit.
_DEG = {"grid2": 4.0, "grid3": 6.0, "geometric": 8.0, "matchings": 6.0, "mix": 6.0}
_FILL = {"grid2": 4.4, "grid3": 7.9, "geometric": 5.7, "matchings": 15.0, "mix": 5.0}


def work(case):
    """One pass reads the Laplacian and the factor once in every iteration (an
    iteration needs all of the one before it) and reads and writes x, r and p."""
    if case["graph"] == "mix":
        count, side = _dims(case)
        n = count * (side / 2 + 16) ** 2
    else:
        n = math.prod(_dims(case))
    cols = _columns(case)
    v = 4 if case["precision"] == "mixed" else 8
    lap, fac = n * (_DEG[case["graph"]] + 1), n * _FILL[case["graph"]]
    if case["entry"] == "apply":
        return {"bytes": fac * (4 + v) + 16 * n, "flops": 4 * fac}
    its = max(1, round(3.75 * -math.log10(case["tol"])))
    return {"bytes": its * ((lap + fac) * (4 + v) + 6 * v * n * cols), "flops": its * cols * (2 * lap + 4 * fac + 12 * n)}


# ---- the same in plain 64-bit torch -------------------------------------------

def _pinv_solve(graphs, b):
    """x with L x = b and zero mean on every graph: Jacobi-preconditioned
    conjugate gradients in FP64 on the block-diagonal Laplacian, refined on the
    true residual.  b: columns x vertices."""
    dev = b.device
    rows, cols, vals, at, comp = [], [], [], 0, []
    for g, a in enumerate(graphs):
        n, m = a.shape[0], a.indices.shape[0]
        j = np.repeat(np.arange(n), np.diff(a.indptr)) + at
        i = a.indices.astype(np.int64) + at
        rows.append(i)
        cols.append(j)
        vals.append(-a.data)
        comp.append(np.full(n, g))
        at += n
        del m
    i, j, w = (np.concatenate(v) for v in (rows, cols, vals))
    d = -np.bincount(j, weights=w, minlength=at)
    i, j, w = np.concatenate([i, np.arange(at)]), np.concatenate([j, np.arange(at)]), np.concatenate([w, d])
    order = np.lexsort((j, i))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=at))])
    L = torch.sparse_csr_tensor(torch.from_numpy(ptr), torch.from_numpy(j[order]), torch.from_numpy(w[order]),
                                size=(at, at), dtype=torch.float64).to(dev)
    dinv = torch.from_numpy(1.0 / d).to(dev)[:, None]
    seg = torch.from_numpy(np.concatenate(comp)).to(dev)
    count = torch.bincount(seg, minlength=len(graphs)).double()[:, None]

    def centred(v):
        if len(graphs) == 1:
            return v - v.mean(dim=0, keepdim=True)
        s = torch.zeros((len(graphs), v.shape[1]), device=dev, dtype=torch.float64).index_add_(0, seg, v)
        return v - (s / count)[seg]

    B = centred(b.T.contiguous())
    x = torch.zeros_like(B)
    for tol in (1e-9, 1e-6, 1e-3):
        r = centred(B - L @ x)
        nr0 = r.norm(dim=0).clamp_min(1e-300)
        e = torch.zeros_like(r)
        z = r * dinv
        p, rho = z.clone(), (r * z).sum(0)
        for it in range(20000):
            q = L @ p
            al = rho / (p * q).sum(0).clamp_min(1e-300)
            e += al * p
            r -= al * q
            if it % 25 == 24 and bool((r.norm(dim=0) <= tol * nr0).all()):
                break
            z = r * dinv
            new = (r * z).sum(0)
            p = z + (new / rho.clamp_min(1e-300)) * p
            rho = new
        x = centred(x + e)
    return x.T.contiguous()


def _ldl_apply(f, r):
    """y = LDLinv r by substitution, one column of the factor at a time
    (forward!, the division by d and backward! of the reference), mean removed."""
    y = r.tolist()
    col, ptr, row, val = (f.col - 1).tolist(), (f.colptr - 1).tolist(), (f.rowval - 1).tolist(), f.fval.tolist()
    for ii, i in enumerate(col):
        yi, last = y[i], ptr[ii + 1] - 1
        for e in range(ptr[ii], last):
            y[row[e]] += yi * val[e]
            yi *= 1.0 - val[e]
        y[row[last]] += yi
        y[i] = yi
    y = [v / d if d != 0 else v for v, d in zip(y, f.d.tolist())]
    for ii in range(len(col) - 1, -1, -1):
        i, last = col[ii], ptr[ii + 1] - 1
        yi = y[i] + y[row[last]]
        for e in range(last - 1, ptr[ii] - 1, -1):
            yi = (1.0 - val[e]) * yi + val[e] * y[row[e]]
        y[i] = yi
    y = np.array(y)
    return y - y.mean()


def exact(case, seed):
    b = _rhs(case, seed)
    if case["entry"] == "apply":
        y = _ldl_apply(_handle("solve", *_key(case)).ldli, b[0].cpu().numpy())
        return torch.from_numpy(y).to(b.device)
    x = _pinv_solve(_graph(*_key(case)), b)
    if case["entry"] == "device":
        return x
    host = x.cpu().numpy()
    if case["entry"] == "group":
        cuts = np.cumsum(_sizes(case))[:-1]
        return [p.copy() for p in np.split(host[0], cuts)]
    if case["entry"] == "serve":
        cuts = np.cumsum(_requests(case))[:-1]
        return [np.ascontiguousarray(p.T) for p in np.split(host, cuts)]
    return host[0].copy() if case["rhs"] == 1 else np.ascontiguousarray(host.T)
