"""The direct sweep's forms at the edges of their ranges, against the replay.

- The two-field infection model (every term but motility) on the largest
  plane priced in place (512^2, 2^16 targets a pass) and just past it, where a
  block's unlike copies are gathered: the default choice on both sides.
- Models of 16 and of 17 types, the most whose tables are held in shared
  memory and the least whose are read where they lie, with and without the
  terms past contact, volume and surface.

Every lattice, volume, surface, type and f32 field is the replay's, bit for
bit.
"""

from __future__ import annotations

import os

import numpy as np
import pytest

from glazier_b200.blueprint import CellType, Model, Species, Start
from glazier_b200.workloads import INFECTION_RULE, infection_start
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _default_kernels(monkeypatch):
    for name in list(os.environ):
        if name.startswith("GLAZIER_"):
            monkeypatch.delenv(name)


def _same(gpu, replay, species: int) -> None:
    labels, want = gpu.labels(), replay.labels()
    assert np.array_equal(labels, want), f"{int((labels != want).sum())} sites differ after {gpu.mcs} MCS"
    assert np.array_equal(gpu.volumes(), replay.volumes())
    assert np.array_equal(gpu.surfaces(), replay.surfaces())
    assert np.array_equal(gpu.cell_types(), replay.cell_types())
    for k in range(species):
        assert np.array_equal(gpu.field(k).astype(np.float32), replay.field(k))


@pytest.mark.parametrize("size, kernel", [(512, "direct"), (514, "gathered")])
def test_the_infection_model_either_side_of_the_gathering_size(device, size, kernel):
    start = infection_start(seed=3, size=size, grid=32, immune=64)
    gpu = device.GpuSimulation.from_start(start)
    assert gpu.sweep_kernel == kernel
    replay = ReplayOracle.from_start(start)
    gpu.set_infection(*INFECTION_RULE)
    replay.set_infection(*INFECTION_RULE)
    for chunk in (1, 5):
        gpu.step(chunk)
        replay.step(chunk)
        _same(gpu, replay, 2)
    gpu.close()


@pytest.mark.parametrize("every", [False, True])
@pytest.mark.parametrize("kinds", [16, 17])
def test_tables_in_shared_memory_and_past_it(device, kinds, every, monkeypatch):
    """`kinds` types in all; without the other terms the passes are launched
    one by one, so the same kernel runs with and without them."""
    monkeypatch.setenv("GLAZIER_SWEEP_RESIDENT", "0")
    n = kinds
    contact = [0.0 if a == b == 0 else 8.0 + (a * 7 + b * 7 + a * b) % 9 for a in range(n) for b in range(n)]
    types = [CellType()]
    for t in range(1, n):
        more = dict(target_length=9.0 + t % 3, lambda_length=0.5 * (t % 2), connected=t % 3 == 0,
                    external=(0.1 * t, -0.2, 0.0)) if every else {}
        types.append(CellType(target_volume=60.0 + t, lambda_volume=1.0 + 0.1 * t, target_surface=90.0 + t,
                              lambda_surface=0.02 * (t % 4), **more))
    model = Model(width=70, height=62, contact=contact, types=types, temperature=11.0, neighbour_order=2, seed=9)
    if every:
        model.species = [Species("signal", 0.2, 0.01, 1.0)]
        model.secretion = [[0.02 * t] for t in range(n)]
        model.uptake = [[0.01 * (t % 3)] for t in range(n)]
        model.chemotaxis = [[5.0 * (t % 2)] for t in range(n)]
    start = Start.tiled(model, 8)
    start.set_cell_types(1 + np.arange(start.n_cells) % (n - 1))
    gpu = device.GpuSimulation.from_start(start)
    assert gpu.sweep_kernel == "direct"
    replay = ReplayOracle.from_start(start)
    gpu.step(12)
    replay.step(12)
    _same(gpu, replay, 1 if every else 0)
    gpu.close()
