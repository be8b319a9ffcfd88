"""Warps that stream over runs of several steps, with every term.

A capped grid gives each warp of the streaming form a run of many steps of 128
targets, whose unlike targets short of a whole round of 32 wait in the warp's
queue for the next step. The models of the parity tests (planes and volumes
with length, nematic, motility, drift, chemotaxis, the connectivity veto,
division and death) on one and on three blocks' warps reproduce the replay bit
for bit.
"""

from __future__ import annotations

import os

import numpy as np
import pytest

import test_gpu_parity
import test_gpu_volume_terms
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu

CASES = {**test_gpu_parity.CASES,
         **{f"terms-{name}": (lambda make=make: (make(), 6)) for name, make in test_gpu_volume_terms.CASES.items()}}


@pytest.fixture(autouse=True)
def _default_kernels(monkeypatch):
    for name in list(os.environ):
        if name.startswith("GLAZIER_"):
            monkeypatch.delenv(name)


@pytest.mark.parametrize("ctas", ["1", "3"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_runs_of_many_steps_reproduce_the_replay(device, name, ctas, monkeypatch):
    made, steps = CASES[name]()
    start, fields = made if isinstance(made, tuple) else (made, None)
    monkeypatch.setenv("GLAZIER_SWEEP_DIRECT", "1")
    monkeypatch.setenv("GLAZIER_SWEEP_CLUSTER", "0")
    monkeypatch.setenv("GLAZIER_SWEEP_COMPACT", "1")
    monkeypatch.setenv("GLAZIER_SWEEP_CTAS", ctas)
    gpu = device.GpuSimulation.from_start(start, fields)
    assert gpu.sweep_kernel == "compact"
    replay = ReplayOracle.from_start(start, fields)
    for chunk in (1, steps - 1):
        gpu.step(chunk)
        replay.step(chunk)
        assert gpu.n_labels == replay.n_labels
        assert np.array_equal(gpu.labels(), replay.labels())
        assert np.array_equal(gpu.volumes(), replay.volumes())
        assert np.array_equal(gpu.surfaces(), replay.surfaces())
        assert np.array_equal(gpu.cell_types(), replay.cell_types())
        for k in range(len(start.model.species)):
            assert np.array_equal(gpu.field(k).astype(np.float32), replay.field(k))
    gpu.close()
