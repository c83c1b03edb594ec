"""Groups of small graphs with one block per graph (csrc/acg_gblock.cuh).

Each member is its own PCG, so it must agree with the oracle on the member
alone (iterations within 1, x within 1e-7; mixed: true residual at the
tolerance): members of two vertices, of one chunk of the dot products (2,048)
and one more, of a few levels and of many, more members than SMs, and one
member too large for the blocks, which takes the whole group to the shared
launches.  A solve with a stop rule of its own per call behaves the same.
"""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G
import oracle as O

pytestmark = pytest.mark.gpu


def _small():
    return [G.path_graph(2), G.path_graph(3), G.star_graph(60), G.complete_graph(33), G.random_tree(700, 3),
            G.grid2(32, 64, weights="loguniform", seed=1), G.grid2(683, 3, weights="loguniform", seed=2),
            G.grid3(9, weights="loguniform", seed=3), G.path_plus_matchings(1200, seed=4)]


GROUPS = {
    "small": _small,
    "many": lambda: [G.grid2(8 + i % 13, 9 + i % 7, weights="loguniform", seed=i) for i in range(170)],
    "one_large": lambda: _small() + [G.grid2(150, weights="loguniform", seed=5)],
}


def _rel(x, y):
    return float(np.linalg.norm(x - y) / max(np.linalg.norm(y), 1e-300))


@pytest.mark.parametrize("name", sorted(GROUPS))
def test_members_match_the_oracle(gpu_ok, name):
    graphs = GROUPS[name]()
    acgpu.seed(13)
    factors = [acgpu.approx_chol(a) for a in graphs]
    grp = acgpu.GroupSolver(graphs, factors)
    bs = [np.random.default_rng(i).standard_normal(a.shape[0]) for i, a in enumerate(graphs)]
    bs[0][:] = 0.0  # a zero right-hand side ends at once
    xs = grp(bs, tol=1e-9, maxits=500)
    its = [i.iterations for i in grp.last_info]
    xm = grp(bs, tol=1e-8, maxits=2000, precision="mixed")
    assert not xs[0].any() and grp.last_info[0].status == 0
    for i, (a, f) in enumerate(zip(graphs, factors)):
        if i == 0 or (name == "many" and i % 17):
            continue
        xo, ito, _, _ = O.OracleSolver(a, f)(bs[i], tol=1e-9, maxits=500)
        assert abs(its[i] - ito) <= 1
        assert _rel(O.center(xs[i]), O.center(xo)) < 1e-7
        assert O.relres(a, xm[i], bs[i] - bs[i].mean()) <= 1e-8 * 1.01
    assert all(np.array_equal(p, q) for p, q in zip(xs, grp(bs, tol=1e-9, maxits=500)))
    for maxits in (0, 1, 10):
        grp(bs, tol=1e-14, maxits=maxits)
        assert all(i.iterations <= maxits for i in grp.last_info)
    grp.close()
