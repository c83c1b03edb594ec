"""A one-vector solve that stops before its first step returns x = 0, in every form
of the solve (csrc/acg_persist.cuh: W for the whole graph, sweeps and tail; and
the per-level engine)."""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1", [20, 60])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("options", [None, dict(sweep_lanes=1)])
def test_no_step_no_x(gpu_ok, n1, precision, options):
    a = G.grid2(n1, weights="loguniform", seed=6)
    acgpu.seed(12)
    dev = acgpu.DeviceLapSolver(a, acgpu.approx_chol(a), options=options)
    b = np.random.default_rng(3).standard_normal(a.shape[0])
    dev(b, tol=1e-9, precision=precision)  # the vectors hold a solve's values
    x = dev(b, tol=1e-9, maxits=0, precision=precision)
    info = dev.last_info[0]
    assert info.iterations == 0 and info.status == 1
    assert not x.any()
    dev.close()
