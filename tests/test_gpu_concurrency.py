"""One-vector solves leave the GPU to other streams (csrc/acg_persist.cuh).

The persistent grid holds nearly all registers of every SM, so its launches end
after a millisecond and the solve's loop starts the next.
"""
import threading
import time

import numpy as np
import pytest

import acgpu
from acgpu import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_other_work_runs_beside_a_long_solve(gpu_ok, precision):
    """Matrix products on another stream, which need free SMs, while a solve of
    many milliseconds runs.  They wait for a pause of the solve (one a
    millisecond), not for its end: without pauses each product took as long as an
    FP64 solve, and one beside a mixed solve half of the longest inner solve.  And
    the solve's result is that of a solve alone, bit for bit."""
    import torch
    a = G.grid3(60, weights="loguniform", seed=1)
    acgpu.seed(1)
    dev = acgpu.DeviceLapSolver(a, acgpu.approx_chol(a))
    b = np.random.default_rng(1).standard_normal(a.shape[0])
    kw = dict(tol=1e-300, maxits=3000, precision=precision)  # until it stagnates
    alone = dev(b, **kw)
    stream = torch.cuda.Stream()
    m = torch.randn(2048, 2048, device="cuda")
    with torch.cuda.stream(stream):
        torch.mm(m, m)
    stream.synchronize()
    out = []

    def work():
        for _ in range(6):
            out.append((dev(b, **kw), dev.last_info[0].solve_ms))

    thread = threading.Thread(target=work)
    thread.start()
    waits = []
    while thread.is_alive():
        t = time.perf_counter()
        with torch.cuda.stream(stream):
            torch.mm(m, m)
        stream.synchronize()
        waits.append(1e3 * (time.perf_counter() - t))
    thread.join()
    assert all(np.array_equal(x, alone) for x, _ in out)
    solve = np.median([ms for _, ms in out])
    assert solve > 8.0
    if precision == "fp64":
        assert np.median(waits) < solve / 8 + 1.0
    else:
        assert max(waits) < solve / 4
    dev.close()
