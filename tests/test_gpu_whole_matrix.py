"""The preconditioner of small graphs as one matrix W (csrc/acg_persist.cuh,
k_form_w): y = W r against substitution in long double.

With W's entries off by at most u |W| + K u^2 (a compensated sum, rounded once), a
row's product (K products on 128 partial sums, joined in 7 additions) is off by at
most (K / 128 + 9) u sum_j |W_ij r_j|, and the mean of y taken out adds the mean of
that and u |y|.  Sums without their errors carried along may be off by another
K u sum_j |W_ij r_j|, 50 times as much at 700 vertices, but are so only in the
worst case, so the kernel's arithmetic is checked in the source too: a product
contracted into the additions would count its rounding error twice.
"""
import pathlib
import re

import numpy as np
import pytest

import acgpu
from acgpu import generators as G

SRC = pathlib.Path(__file__).parents[1] / "laplacians.jl_b200" / "csrc" / "acg_persist.cuh"
U = 2.0 ** -53


def test_the_compensated_sum_is_not_contracted():
    body = SRC.read_text().split("k_form_w(int K")[1]
    loop = body[body.index("#pragma unroll 4"):body.index("acc[a][b] = sum;")]
    names = r"(?:prod|sum|old|low\[a\]\[b\]|err|\bt\b|\bx\b|\bz\b)"
    assert not re.search(names + r"\s*[*+]=?\s*" + names, loop)
    assert not re.search(names + r"\s*-\s*" + names, loop)
    for op in ("__dmul_rn", "__dadd_rn", "__dsub_rn", "__fma_rn"):
        assert op in loop


def _operator(f, n):
    """M^T diag(g) M of the factor, dense, in long double: its columns are the
    substitutions of unit vectors."""
    one = np.longdouble(1)
    y = np.eye(n, dtype=np.longdouble)
    col, ptr, row, val = f.col - 1, f.colptr - 1, f.rowval - 1, f.fval.astype(np.longdouble)
    for ii, i in enumerate(col):
        last = ptr[ii + 1] - 1
        yi = y[i].copy()
        for e in range(ptr[ii], last):
            y[row[e]] += yi * val[e]
            yi = yi * (one - val[e])
        y[row[last]] += yi
        y[i] = yi
    d = f.d.astype(np.longdouble)
    y = np.where((d != 0)[:, None], y / np.where(d != 0, d, one)[:, None], y)
    for ii in range(len(col) - 1, -1, -1):
        i, last = col[ii], ptr[ii + 1] - 1
        yi = y[i] + y[row[last]]
        for e in range(last - 1, ptr[ii] - 1, -1):
            yi = (one - val[e]) * yi + val[e] * y[row[e]]
        y[i] = yi
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["grid2", "matchings", "path", "grid3"])
def test_w_against_long_double(gpu_ok, name):
    a = {"grid2": lambda: G.grid2(26, 27, weights="loguniform", seed=1),
         "matchings": lambda: G.path_plus_matchings(700, sigma=2.0, seed=2),
         "path": lambda: G.path_graph(650), "grid3": lambda: G.grid3(9, weights="lognormal:2", seed=3)}[name]()
    n = a.shape[0]
    acgpu.seed(3)
    f = acgpu.approx_chol(a)
    w = _operator(f, n)
    # what k_form_w leaves out shifts y by a constant: each column's mean over the
    # rows but for terms in the mean of r (zero here), so the centred operator
    # bounds its entries from below; the kernel's own are bounded by twice the
    # largest distance of a column's entries from their mean
    c = w - w.mean(axis=0)
    size = 2 * np.abs(c).max(axis=0)
    dev = acgpu.DeviceLapSolver(a, f)
    for seed in range(3):
        r = np.random.default_rng(seed).standard_normal(n)
        r -= r.mean()
        y = c @ r.astype(np.longdouble)
        y -= y.mean()
        bound = 2 * (n / 128 + 9) * U * float(size @ np.abs(r)) + 2 * U * np.abs(y).max()
        assert np.abs(dev.ldlsolve(r) - y).max() <= bound
    dev.close()
