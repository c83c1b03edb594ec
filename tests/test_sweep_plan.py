"""The sweep plan (csrc/acg_plan.h) on the host, without a GPU.

plan_check.cpp is compiled with the plan's source into a temporary library; the
plans are built for factors of the host elimination and for DAGs made here, and
their rows are walked in plain numpy.
"""
import ctypes
import pathlib
import subprocess
import sys

import numpy as np
import pytest

import acgpu
from acgpu import generators as G

HERE = pathlib.Path(__file__).parent
CSRC = HERE.parent / "laplacians.jl_b200" / "csrc"
VECTOR = (25000.0, 128.0, 0.4, 160, 64, 3.0, 2 << 20)  # kVectorCost, kBatchCost
BATCH = (10000.0, 32.0, 0.5, 0, 0, 2.0, 1 << 20)
PART = 3  # kRowPart


@pytest.fixture(scope="session")
def lib_path(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "plan_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC,
                    HERE / "plan_check.cpp", CSRC / "acg_plan.cpp", "-o", out, "-lpthread"], check=True)
    return out


class Dag:
    """CSR of the in-edges (ascending) and of the column entries (descending);
    `levels`: per level one vertex range per graph."""

    def __init__(self, n, levels, dst, src, val, tail=None):
        self.n, self.levels = n, levels
        self.tail = len(levels) if tail is None else tail
        o = np.lexsort((src, dst))
        self.fptr = np.concatenate([[0], np.cumsum(np.bincount(dst, minlength=n))]).astype(np.int32)
        self.fidx, self.fc = src[o].astype(np.int32), val[o].astype(np.float64)
        o = np.lexsort((-dst, src))
        self.bptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
        self.bidx, self.bc = dst[o].astype(np.int32), val[o].astype(np.float64)

    def build(self, path, cost, merge=True, fail=False):
        lib = ctypes.CDLL(str(path))
        lib.pc_build.restype = ctypes.c_void_p
        runs = np.array([(i, a, b) for i, lv in enumerate(self.levels) for a, b in lv], np.int32)

        def c(a):
            return ctypes.c_void_p(a.ctypes.data)

        cst = np.array(cost, np.float64)
        h = lib.pc_build(self.n, len(self.levels), len(runs), c(runs), c(self.fptr), c(self.fidx), c(self.fc),
                         c(self.bptr), c(self.bidx), c(self.bc), self.tail, c(cst), int(merge), int(fail))
        if not h:
            return None
        h = ctypes.c_void_p(h)
        dims = np.zeros(8, np.int64)
        lib.pc_dims(h, c(dims))
        out = {"slots": int(dims[0]), "blocks": int(dims[1])}
        for d, name in enumerate(("fwd", "bwd")):
            nr, rows, nnz = (int(v) for v in dims[2 + 3 * d:5 + 3 * d])
            r, p, i, v = (np.empty((nr, 5), np.int32), np.empty(rows + 1, np.int32), np.empty(nnz, np.int32),
                          np.empty(nnz, np.float64))
            lib.pc_rows(h, d, c(r), c(p), c(i), c(v))
            out[name] = (r, p, i, v)
        lib.pc_free(h)
        return out


def layers(nlev, width, seed=0, fan=3):
    """nlev levels of `width` vertices, each with `fan` inputs one level down."""
    rng = np.random.default_rng(seed)
    n = nlev * width
    dst = np.repeat(np.arange(width, n), fan)
    src = (dst // width - 1) * width + rng.integers(0, width, dst.shape[0])
    pair = np.unique(np.stack([dst, src]), axis=1)
    return Dag(n, [[(i * width, (i + 1) * width)] for i in range(nlev)], pair[0], pair[1],
               rng.uniform(0.1, 0.3, pair.shape[1]))


def test_a_run_of_rows_belongs_to_one_graph(lib_path):
    """A group's task tables are cut by graph, so no run may hold rows of two: a
    graph without factor entries (one level) lies next to the first level of the
    one after it."""
    # graph 0: vertices 0 and 1, no entries; graph 1: vertices 2 and 3, then 4
    dag = Dag(5, [[(0, 2), (2, 4)], [(4, 5)]], np.array([4, 4]), np.array([2, 3]), np.array([0.5, 0.5]))
    plan = dag.build(lib_path, VECTOR, merge=False)
    for name in ("fwd", "bwd"):
        for v0, count, *_ in plan[name][0]:
            assert (v0 < 2) == (v0 + count - 1 < 2)


def factor_dag(a, seed=1, dense_tail=2048):
    """The DAG of a graph's factor, numbered as the solver numbers it: by level,
    then by falling in-degree, then by elimination step; coefficients folded.
    Also the plain factor's in-edges (the oracle of the sweeps)."""
    acgpu.seed(seed)
    f = acgpu.approx_chol(a)
    n = a.shape[0]
    col, ptr, row = f.col - 1, f.colptr - 1, f.rowval - 1
    src = np.repeat(col, np.diff(ptr))
    step = np.full(n, n - 1)
    step[col] = np.arange(n - 1)
    lev = np.zeros(n, np.int64)
    val = np.empty(f.fval.shape[0])
    for i, u in enumerate(col):
        e = slice(ptr[i], ptr[i + 1])
        lev[row[e]] = np.maximum(lev[row[e]], lev[u] + 1)
        left = np.concatenate([[1.0], np.cumprod(1.0 - f.fval[e][:-1])])
        val[e] = left * np.append(f.fval[e][:-1], 1.0)
    indeg = np.bincount(row, minlength=n)
    perm = np.lexsort((step, -indeg, lev))
    num = np.empty(n, np.int64)
    num[perm] = np.arange(n)
    off = np.concatenate([[0], np.cumsum(np.bincount(lev))])
    levels = [[(int(off[i]), int(off[i + 1]))] for i in range(len(off) - 1)]
    tail = len(levels)
    while tail > 0 and n - off[tail - 1] <= min(dense_tail, n // 4):
        tail -= 1
    if len(levels) - tail < 8:
        tail = len(levels)
    dst, s = num[row], num[src]
    v0 = off[tail] if tail < len(levels) else n
    keep = ~((dst >= v0) & (s >= v0))  # the sweeps keep the tail's inputs from the head
    d = Dag(n, levels, dst[keep], s[keep], val[keep], tail)
    full = Dag(n, levels, dst, s, val)
    d.bptr, d.bidx, d.bc = full.bptr, full.bidx, full.bc
    return d


GRAPHS = {
    "path2": lambda: G.path_graph(2), "path3000": lambda: G.path_graph(3000), "star2000": lambda: G.star_graph(2000),
    "tree4000": lambda: G.random_tree(4000, 4), "complete60": lambda: G.complete_graph(60),
    "grid2_61x47": lambda: G.grid2(61, 47, weights="loguniform", seed=2),
    "grid3_17": lambda: G.grid3(17, weights="loguniform", seed=3),
    "matchings6000": lambda: G.path_plus_matchings(6000, seed=5),
}


def walk(plan, name, term, given):
    """The plan's rows in their order, `term` a vertex's own term: every slot is
    written once, and none is read before.  `given`: values there from the start
    (NaN: none)."""
    runs, ptr, idx, coef = plan[name]
    out = np.full(plan["slots"], np.nan)
    out[:given.shape[0]] = given
    for v0, count, kind, delta, row in runs:
        for i in range(count):
            e = slice(ptr[row + i], ptr[row + i + 1])
            total = float(coef[e] @ out[idx[e]]) + (term[v0 + i] if kind in (0, 1) else 0.0)
            slot = v0 + i + (delta if kind in (1, PART) else 0)
            assert np.isnan(out[slot]) and not np.isnan(total)
            out[slot] = total
    return out[:given.shape[0]]


@pytest.mark.parametrize("cost,merge", [(VECTOR, True), (VECTOR[:3] + (16, 5) + VECTOR[5:], True), (BATCH, True),
                                        (VECTOR, False)])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_the_rows_are_the_substitutions(lib_path, name, cost, merge):
    """Both directions against plain substitution over the DAG, to 1e-13 of the
    largest value (a row sums at most a few thousand non-negative products)."""
    d = factor_dag(GRAPHS[name]())
    plan = d.build(lib_path, cost, merge)
    rng = np.random.default_rng(1)
    r, g = rng.uniform(0.5, 1.5, d.n), rng.uniform(0.5, 1.5, d.n)
    v0 = d.levels[d.tail][0][0] if d.tail < len(d.levels) else d.n
    s = r.copy()
    for v in range(d.n):
        e = slice(d.fptr[v], d.fptr[v + 1])
        s[v] += d.fc[e] @ s[d.fidx[e]]
    none = np.full(d.n, np.nan)
    assert np.abs(walk(plan, "fwd", r, none) - s).max() <= 1e-13 * s.max()
    y = g * s  # the tail's values are given
    none[v0:] = y[v0:]
    for v in range(v0 - 1, -1, -1):
        e = slice(d.bptr[v], d.bptr[v + 1])
        y[v] += d.bc[e] @ y[d.bidx[e]]
    assert np.abs(walk(plan, "bwd", g * s, none) - y).max() <= 1e-13 * y.max()


@pytest.mark.parametrize("cost", [VECTOR, BATCH])
def test_deep_factors_do_not_fill_the_device(lib_path, cost):
    """The blocks' entries stay within the limit however deep the DAG is: a path's
    factor (one entry a column, as many levels as vertices) took 127 entries a
    vertex."""
    d = factor_dag(G.path_graph(60000))
    factor = int(d.bptr[-1])
    lib = ctypes.CDLL(str(lib_path))
    lib.pc_fill_limit.restype = ctypes.c_longlong
    c = np.array(cost, np.float64)
    limit = lib.pc_fill_limit(ctypes.c_void_p(c.ctypes.data), d.n, ctypes.c_longlong(factor))
    assert limit == max(cost[5] * factor, cost[6])
    plan = d.build(lib_path, cost)
    head = d.levels[d.tail][0][0]
    assert plan["blocks"] < head  # still merged
    for name in ("fwd", "bwd"):
        assert len(plan[name][2]) <= (factor + limit) * (1 + 2 / 64)


@pytest.mark.parametrize("cost", [VECTOR, BATCH])
@pytest.mark.parametrize("n,factor", [(10**6, 8 * 10**6), (2 * 10**8, 10**9), (10**9, 10**9), (2 * 10**9, 2 * 10**9),
                                      (10**6, 2**31 - 2), (1000, 2 * 10**9)])
def test_plans_of_large_factors_stay_in_int_range(lib_path, cost, n, factor):
    """Entries, slots and rows of a plan are ints: what a limit other than 0 (no
    merging, no cutting) allows has to fit."""
    lib = ctypes.CDLL(str(lib_path))
    lib.pc_fill_limit.restype = ctypes.c_longlong
    c = np.array(cost, np.float64)
    limit = lib.pc_fill_limit(ctypes.c_void_p(c.ctypes.data), n, ctypes.c_longlong(factor))
    if limit == 0:
        assert factor + n > 10**9
        return
    entries = factor + limit
    parts = -(-entries // cost[4]) + entries // cost[3] if cost[3] else 0
    assert entries + parts < 2**31  # a long row's parts are entries of the row
    assert 2 * n + parts < 2**31    # values, work values, parts; as many rows


def test_an_allocation_that_fails_on_a_thread_is_an_exception(lib_path):
    """The plan of a DAG large enough for several threads, with allocations off the
    calling thread failing: the caller gets std::bad_alloc (the C entries' error
    code) and the process goes on.  In a process of its own, which an unhandled
    exception would end."""
    code = (f"import sys; sys.path[:0] = {sys.path!r}; import test_sweep_plan as t; "
            f"d = t.layers(20, 15000); assert d.build({str(lib_path)!r}, t.VECTOR, fail=True) is None; "
            f"assert d.build({str(lib_path)!r}, t.VECTOR)['blocks'] > 0; print('went on')")
    res = subprocess.run([sys.executable, "-c", code], cwd=HERE, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "went on" in res.stdout, res.stderr[-2000:]
