"""Reductions of the batched iteration (csrc/acg_batch.cuh).

The sums over the grid run in one level while the last block's threads read at
most 8 rows of partials each (blocks times columns <= 2,048), else in two.  Graphs
on both sides of that line, for the mat-vec (32 rows a block) and the vector
kernels (2 KB of a vector per 256 threads and step), at every padded number of
columns, full and ragged: each column takes the oracle's iterations within 1 and
its solution within 1e-7 at tol 1e-9, and a second call gives the same bits.
"""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [2, 8, 9, 16, 31, 64])
@pytest.mark.parametrize("dims", [(3, 5), (16, 32), (23, 23), (64, 64), (91, 90), (183, 180)])
def test_columns_match_the_oracle(gpu_ok, dims, cols):
    a = G.grid2(*dims, weights="loguniform", seed=4)
    acgpu.seed(13)
    ldli = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, ldli)
    orc = O.OracleSolver(a, ldli)
    B = np.random.default_rng(cols).standard_normal((a.shape[0], cols))
    X = dev(B, tol=1e-9, maxits=500)
    info = list(dev.last_info)
    assert np.array_equal(dev(B, tol=1e-9, maxits=500), X)
    for c in sorted({0, cols // 2, cols - 1}):
        xo, ito, _, _ = orc(B[:, c].copy(), tol=1e-9, maxits=500)
        assert abs(info[c].iterations - ito) <= 1
        x = O.center(X[:, c])
        assert np.linalg.norm(x - O.center(xo)) <= 1e-7 * np.linalg.norm(O.center(xo))
    Xm = dev(B, tol=1e-8, maxits=2000, precision="mixed")
    for c in (0, cols - 1):
        b = B[:, c] - B[:, c].mean()
        assert O.relres(a, Xm[:, c], b) <= 1e-8 * 1.01
    dev.close()
