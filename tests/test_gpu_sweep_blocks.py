"""The sweeps' merged blocks of levels (csrc/acg_plan.h).

A block applies M_B = (I - C_BB)^{-1} instead of its levels one by one: the same
operator with another order of rounding, so LDLsolver must agree with the
oracle to 1e-12 relative in FP64 and 1e-4 in FP32 (the bars of the sweep
parity tests) whatever the DAG: chains that become one block, a star's long
row, trees, rows longer than a warp's entries in flight, and with the dense
tail off, where the narrow end of the DAG is merged too.  The batched sweeps
have their own plan; a batch of one column more than a power of two pads.
"""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G
import oracle as O

pytestmark = pytest.mark.gpu

GRAPHS = {
    "path2": lambda: G.path_graph(2),
    "path700": lambda: G.path_graph(700),
    "cycle301": lambda: G.cycle_graph(301),
    "star900": lambda: G.star_graph(900),
    "complete40": lambda: G.complete_graph(40),
    "tree3000": lambda: G.random_tree(3000, 4),
    "grid2_97x31": lambda: G.grid2(97, 31, weights="loguniform", seed=2),
    "grid3_19": lambda: G.grid3(19, weights="loguniform", seed=3),
    "matchings9000": lambda: G.path_plus_matchings(9000, seed=5),
}


def _rel(x, y):
    return float(np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-300))


@pytest.mark.parametrize("tail", [0, -1])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_merged_sweeps_match_the_oracle(gpu_ok, name, tail):
    a = GRAPHS[name]()
    n = a.shape[0]
    acgpu.seed(7)
    ldli = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, ldli, options=dict(dense_tail=tail))
    r = np.random.default_rng(n).standard_normal(n)
    r -= r.mean()
    y_ref = O.ldlsolve(ldli, r)
    y = dev.ldlsolve(r)
    assert _rel(y, y_ref) < 1e-12
    assert _rel(dev.ldlsolve(r, "mixed"), y_ref) < 1e-4
    assert np.array_equal(dev.ldlsolve(r), y)  # no state between calls
    B = np.random.default_rng(n + 1).standard_normal((n, 9))
    X = dev(B, tol=1e-9, maxits=500)
    for c in (0, 8):
        xo, ito, _, _ = O.OracleSolver(a, ldli)(B[:, c], tol=1e-9, maxits=500)
        assert abs(dev.last_info[c].iterations - ito) <= 1
        assert _rel(O.center(X[:, c]), O.center(xo)) < 1e-7
    dev.close()
