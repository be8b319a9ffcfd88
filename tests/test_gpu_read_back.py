"""Read-backs into pinned memory take as long as the copy.

A pinned buffer has its pages, so nothing is done to them before the copy. The
time is held to torch's own copy of the same bytes: at 64 MB the walk through
the buffer's pages that a pageable buffer's read-back begins with would make
it 1.4 times that.
"""

from __future__ import annotations

import time

import numpy as np
import pytest

from glazier_b200.workloads import monolayer

pytestmark = pytest.mark.gpu


def _least(f, times: int) -> float:
    best = float("inf")
    for _ in range(times):
        t0 = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t0)
    return best


def test_a_pinned_buffer_is_filled_at_the_copy_rate(device):
    import torch

    start = monolayer(4096)
    with device.GpuSimulation.from_start(start) as sim:
        sim.step(1)
        pinned = torch.zeros(sim.sites, dtype=torch.int32).pin_memory()
        source = torch.zeros(sim.sites, dtype=torch.int32, device="cuda")

        def plain():
            pinned.copy_(source)
            torch.cuda.synchronize()

        def read():
            sim.labels_to(pinned.data_ptr(), sim.sites)

        plain(), read()
        # 1.2: half way to the walk's cost, far past what either time varies by
        assert _least(read, 30) < 1.2 * _least(plain, 30)
        read()
        assert np.array_equal(pinned.numpy().view(np.uint32), sim.labels())
        # a buffer that does not start on a page, and one of a few sites more
        out = np.zeros(sim.sites + 3, dtype=np.uint32)
        sim.labels_into(out[1:-2])
        assert np.array_equal(out[1:-2], sim.labels()) and out[0] == 0 and not out[-2:].any()
