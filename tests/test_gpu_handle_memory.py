"""What a handle holds on the device, and when."""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G

pytestmark = pytest.mark.gpu


def test_the_batched_plan_comes_with_the_first_batch(gpu_ok):
    """A handle that solves single vectors holds no plan for batches.  The first
    batch of 8 columns adds the plan to the batch buffers, a batch of 16 doubles
    the buffers alone, so the first growth is larger by the plan: 16 bytes an entry
    (an index, two value types) in each direction, of at least half the factor's
    entries (the dense tail's substitutions are not swept)."""
    a = G.grid3(30, weights="loguniform", seed=2)
    acgpu.seed(3)
    f = acgpu.approx_chol(a)
    dev = acgpu.DeviceLapSolver(a, f)
    B = np.random.default_rng(1).standard_normal((a.shape[0], 16))
    x = dev(B[:, 0], tol=1e-9)
    held = [dev.stats()["device_bytes"]]
    for k in (8, 16):
        X = dev(B[:, :k], tol=1e-9)
        held.append(dev.stats()["device_bytes"])
        assert np.linalg.norm(X[:, 0] - x) <= 1e-7 * np.linalg.norm(x)
    first, second = held[1] - held[0], held[2] - held[1]
    assert first - second > 16 * f.nnz  # the reductions' partial sums alone are 1.2 MB of 3.4
    dev.close()
