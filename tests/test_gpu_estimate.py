"""SolveServer's estimate of what a graph holds on the device against what the
driver says: at least as much, so that the budget holds, and not many times it."""
import numpy as np
import pytest

import acgpu
from acgpu import generators as G
from acgpu.serving import SolveServer, _GraphEntry

pytestmark = pytest.mark.gpu

GRAPHS = {
    "grid2_20": lambda: G.grid2(20, weights="loguniform", seed=1),
    "grid2_45": lambda: G.grid2(45, weights="loguniform", seed=1),
    "path9000": lambda: G.path_graph(9000),
    "matchings20000": lambda: G.path_plus_matchings(20000, sigma=2.0, seed=1),
    "grid3_50": lambda: G.grid3(50, weights="loguniform", seed=1),
}


@pytest.mark.parametrize("slots", [8, 64])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_the_estimate_covers_a_served_graph(gpu_ok, name, slots):
    import torch
    a = GRAPHS[name]()
    acgpu.seed(1)
    f = acgpu.approx_chol(a)
    server = SolveServer(1 << 40, slots=slots)
    est = server._estimate_bytes(_GraphEntry("x", a, f))
    held = 0
    for i in range(2):  # the first may load kernels
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        dev = acgpu.DeviceLapSolver(a, f)
        loop = acgpu.ServeLoop(dev, precision="mixed", slots=server.slots, queue=server.queue)
        b = np.random.default_rng(1).standard_normal((a.shape[0], 2))
        loop.submit(b, tol=1e-6).wait()
        dev(b[:, 0], tol=1e-6)
        torch.cuda.synchronize()
        held = before - torch.cuda.mem_get_info()[0]
        loop.close()
        dev.close()
    # the driver hands memory out in 2 MB pieces, and keeps some for the graphs
    assert held <= est + (96 << 20)
    assert est <= 8 * held + (256 << 20)
