"""Both forms of a group's solve (csrc/acg_group.cuh and csrc/acg_gblock.cuh) give
the same bits, whatever the sizes: members on both sides of what the swept vector
and p need in a block's shared memory (about 28,000 and 14,000 FP64 values, twice
as many FP32 ones), members of one chunk of the dot products and more, and more
members than SMs.  A group under the rule gives the bits of both.
"""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G

pytestmark = pytest.mark.gpu

SHARED, BLOCKS = dict(sweep_lanes=2), dict(sweep_lanes=3)
GROUPS = {
    "small": lambda: [G.path_graph(2), G.star_graph(60), G.grid2(32, 64, weights="loguniform", seed=1),
                      G.grid2(683, 3, weights="loguniform", seed=2), G.path_plus_matchings(3000, seed=4)],
    "p_in_global": lambda: [G.grid2(127, 128, weights="loguniform", seed=1), G.grid2(20, weights="loguniform", seed=2)],
    "v_in_global": lambda: [G.grid2(180, 181, weights="loguniform", seed=1), G.grid2(250, 251, weights="loguniform", seed=2),
                            G.grid3(8, weights="loguniform", seed=3)],
    "many": lambda: [G.grid2(8 + i % 13, 9 + i % 7, weights="loguniform", seed=i) for i in range(170)],
}


@pytest.mark.parametrize("name", sorted(GROUPS))
def test_both_forms_give_the_same_bits(gpu_ok, name):
    graphs = GROUPS[name]()
    acgpu.seed(13)
    factors = [acgpu.approx_chol(a) for a in graphs]
    bs = [np.random.default_rng(i).standard_normal(a.shape[0]) for i, a in enumerate(graphs)]
    out = []
    for options in (SHARED, BLOCKS, None):
        grp = acgpu.GroupSolver(graphs, factors, options=options)
        runs = []
        for kw in (dict(tol=1e-9, maxits=400), dict(tol=1e-14, maxits=11),
                   dict(tol=1e-8, maxits=2000, precision="mixed")):
            xs = grp(bs, **kw)
            runs.append((xs, [(i.iterations, i.status) for i in grp.last_info]))
        grp.close()
        out.append(runs)
    for other in out[1:]:
        for (xs, info), (ys, jnfo) in zip(out[0], other):
            assert info == jnfo
            assert all(np.array_equal(x, y) for x, y in zip(xs, ys))
