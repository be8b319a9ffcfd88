"""What an engine waits for, and on which stream.

An engine is set up on its own stream: with a second of another user's work
queued on the default stream, an engine with every uploaded array (fields,
nematic field, activity and its list of accepted copies) is made and stepped
before that work ends, and the run is the replay's.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import sheet_model, tiled, with_species
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu


def test_the_default_stream_is_not_waited_for(device):
    import torch

    model = with_species(sheet_model(width=96, height=64, seed=17, max_activity=20.0, lambda_activity=60.0,
                                     lambda_nematic=3.0),
                         [("a", 0.2, 0.01, 1.0), ("b", 0.1, 0.0, 0.5)], [[0.0, 0.0], [0.2, 0.1]],
                         [[0.0, 0.0], [0.01, 0.0]], [[0.0, 0.0], [3.0, 0.0]])
    model.nematic = np.random.default_rng(19).uniform(-0.5, 0.5, size=(model.sites, 2))
    start = tiled(model, 8, 10, 7)
    replay = ReplayOracle.from_start(start)
    replay.step(10)
    with device.GpuSimulation.from_start(start) as warm:  # the library's kernels are loaded
        warm.step(1)
        warm.labels(), warm.field(0)
    other = torch.cuda.default_stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000_000)  # about a second of the default stream
    sim = device.GpuSimulation.from_start(start)
    sim.step(10)
    assert not other.query(), "the engine waited for the default stream"
    assert np.array_equal(sim.labels(), replay.labels())
    for k in range(2):
        assert np.array_equal(sim.field(k).astype(np.float32), replay.field(k))
    torch.cuda.synchronize()
    sim.close()


def test_no_steps_wait_for_nothing(device):
    """A call of no steps returns with its stream's earlier work still queued."""
    import torch

    with device.GpuSimulation.from_start(tiled(sheet_model(seed=3))) as sim:
        before = sim.labels()
        own = torch.cuda.ExternalStream(sim.stream)
        with torch.cuda.stream(own):
            torch.cuda._sleep(400_000_000)  # about a fifth of a second
        sim.step(0)
        assert sim.step_profiled(0) == (0.0, 0.0, 0.0)
        assert not own.query(), "a call of no steps waited"
        own.synchronize()
        assert sim.mcs == 0 and np.array_equal(sim.labels(), before)
