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


def test_a_closed_handle_gives_its_memory_back(gpu_ok):
    """Twelve handles opened, used in every way that allocates and closed one after
    another: the device has as much free memory afterwards as after the first two,
    up to 64 MB that the driver may keep (each holds more than 100 MB)."""
    import torch
    a = G.grid2(150, weights="loguniform", seed=2)
    acgpu.seed(3)
    f = acgpu.approx_chol(a)
    small = [G.grid2(20), G.grid2(30)]
    B = np.random.default_rng(1).standard_normal((a.shape[0], 64))
    free = []
    for i in range(12):
        dev = acgpu.DeviceLapSolver(a, f)
        dev(B[:, 0], tol=1e-2)
        dev(B, tol=1e-2)
        dev.solve_async(B, tol=1e-2).wait()
        assert dev.stats()["device_bytes"] > 100 << 20
        dev.close()
        g = acgpu.GroupSolver(small)
        g([B[:400, 0], B[:900, 0]], tol=1e-2)
        g.close()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[-1] <= 64 << 20


def test_a_handle_closed_before_its_tickets_are_waited(gpu_ok):
    """acg_destroy serves the requests that a loop holds before anything is freed;
    their tickets give the solutions afterwards."""
    a = G.grid3(20, weights="loguniform", seed=2)
    acgpu.seed(3)
    dev = acgpu.DeviceLapSolver(a, acgpu.approx_chol(a))
    b = np.random.default_rng(1).standard_normal((a.shape[0], 3))
    x = dev(b, tol=1e-9, precision="mixed")
    loop = acgpu.ServeLoop(dev, precision="mixed", slots=8)
    tickets = [loop.submit(b[:, c], tol=1e-9) for c in range(3)]
    dev.close()
    for c, t in enumerate(tickets):
        assert np.linalg.norm(t.wait() - x[:, c]) <= 1e-6 * np.linalg.norm(x[:, c])
    loop._h = None  # closed with its solver
