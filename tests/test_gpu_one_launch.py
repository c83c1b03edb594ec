"""One-vector solves as one persistent launch (csrc/acg_persist.cuh).

The PCG is the reference's, so iteration counts and solutions must be the
oracle's as in the parity tests (iterations within 1, x within 1e-7) at the
sizes where the launch changes form: the smallest graph, up to 2,048 vertices
(the whole preconditioner as one symmetric matrix), one vertex more, sizes
around the padding of its rows and of the dense tail, and no dense tail at
all.  Stop rules act as in the launch-per-kernel form of the per-level engine.
"""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G
import oracle as O

pytestmark = pytest.mark.gpu

GRAPHS = {
    "path2": lambda: G.path_graph(2),
    "path63": lambda: G.path_graph(63),
    "grid2_8x8": lambda: G.grid2(8),
    "grid2_5x13": lambda: G.grid2(5, 13, weights="loguniform", seed=1),
    "grid2_32x64": lambda: G.grid2(32, 64, weights="loguniform", seed=2),  # 2,048
    "grid2_683x3": lambda: G.grid2(683, 3, weights="loguniform", seed=3),  # 2,049
    "grid3_16": lambda: G.grid3(16, weights="loguniform", seed=4),
    "matchings9001": lambda: G.path_plus_matchings(9001, seed=5),
}


def _rel(x, y):
    return float(np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-300))


@pytest.mark.parametrize("tail", [0, -1])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_solves_match_the_oracle(gpu_ok, name, tail):
    a = GRAPHS[name]()
    n = a.shape[0]
    acgpu.seed(11)
    ldli = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, ldli, options=dict(dense_tail=tail))
    orc = O.OracleSolver(a, ldli)
    for seed in (1, 2):
        b = np.random.default_rng(seed).standard_normal(n)
        x = dev(b, tol=1e-9, maxits=500)
        xo, ito, _, _ = orc(b, tol=1e-9, maxits=500)
        assert abs(dev.last_info[0].iterations - ito) <= 1
        assert _rel(O.center(x), O.center(xo)) < 1e-7
        assert np.array_equal(dev(b, tol=1e-9, maxits=500), x)  # the same bits again
        xm = dev(b, tol=1e-8, maxits=2000, precision="mixed")
        assert O.relres(a, xm, b - b.mean()) <= 1e-8 * 1.01
    dev.close()


@pytest.mark.parametrize("n1", [20, 60])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stop_rules_match_the_per_level_engine(gpu_ok, n1, precision):
    a = G.grid2(n1, weights="loguniform", seed=6)
    acgpu.seed(12)
    ldli = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, ldli)
    ref = acgpu.DeviceLapSolver(a, ldli, options=dict(sweep_lanes=1))
    b = np.random.default_rng(3).standard_normal(a.shape[0])
    for kw in (dict(maxits=0), dict(maxits=1), dict(maxits=9), dict(maxits=10), dict(maxits=11), dict(tol=1e-1)):
        kw = dict(dict(tol=1e-12), **kw)
        x, y = dev(b, precision=precision, **kw), ref(b, precision=precision, **kw)
        i, j = dev.last_info[0], ref.last_info[0]
        assert (i.status, i.iterations) == (j.status, j.iterations), kw
        assert _rel(x, y) < 1e-4 or not y.any()
    dev(b, tol=1e-12, maxtime=0.0)
    assert dev.last_info[0].status == 7  # maxtime
    z = dev(np.zeros(a.shape[0]), precision=precision)
    assert dev.last_info[0].status == 0 and not z.any()
    dev.close()
    ref.close()
