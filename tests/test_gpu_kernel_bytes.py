"""acg_time_kernels counts the bytes of the factor, not those of the sweep plan: what
the merged levels add is no work that a solve cannot do without."""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,vb", [("fp64", 8), ("mixed", 4)])
def test_sweep_bytes_are_the_factors(gpu_ok, precision, vb):
    a = G.grid3(20, weights="loguniform", seed=2)
    n = a.shape[0]
    acgpu.seed(3)
    f = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, f, options=dict(dense_tail=-1))
    dev(np.random.default_rng(1).standard_normal(n), tol=1e-2)
    rows = f.nnz * (4 + vb) + 4 * (n + 1)
    one, many = dev.time_kernels(precision, reps=2), dev.time_kernels_batch(16, precision, reps=2)
    assert one["forward_sweep_bytes"] == rows + 3 * n * vb
    assert one["backward_sweep_bytes"] == rows + 4 * n * vb
    assert many["forward_sweep_bytes"] == rows + 3 * n * 16 * vb
    assert many["backward_sweep_bytes"] == rows + n * vb + 3 * n * 16 * vb
    dev.close()
