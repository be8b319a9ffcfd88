"""Targets of terms that a model does not have, against the replay.

A type whose volume or surface weight is zero has no such term, whatever
target stands beside it: infinite, NaN, so large that twice its distance
leaves f32, or past f32 altogether. The medium has neither term, although its
table entry is its first cell type's, so an infinite target with a weight
changes that type's cells alone. Every sweep kernel and the ensemble price
these the replay's way, bit for bit.
"""

from __future__ import annotations

import math
import os

import numpy as np
import pytest

from glazier_b200.blueprint import CellType, Model, Start
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu

KERNELS = {
    "cluster": {"RESIDENT": "1"},
    "direct": {"DIRECT": "1", "COMPACT": "0", "CLUSTER": "0"},
    "compact": {"DIRECT": "1", "COMPACT": "1", "CLUSTER": "0"},
    "gathered": {"DIRECT": "1", "COMPACT": "2", "CLUSTER": "0"},
    "lean": {"DIRECT": "0"},
    "general": {"DIRECT": "0", "LEAN": "0"},
    "band": {"BAND": "1"},
}


@pytest.fixture(autouse=True)
def _default_kernels(monkeypatch):
    for name in list(os.environ):
        if name.startswith("GLAZIER_"):
            monkeypatch.delenv(name)


def _start(types: int, target: float, term: str, weighted: bool, seed: int = 11) -> Start:
    """Cells of side 8 in a 64 x 64 plane with medium around them; with
    `weighted` the first type carries the target with a weight."""
    cell = dict(target_volume=64.0, lambda_volume=1.0, target_surface=90.0, lambda_surface=0.05)
    odd = dict(cell)
    odd[f"target_{term}"] = target
    odd[f"lambda_{term}"] = 0.5 if weighted else 0.0
    model = Model(width=64, height=64, contact=[0.0, 16.0, 16.0, 16.0, 6.0, 10.25, 16.0, 10.25, 9.125],
                  types=[CellType(), CellType(**odd), CellType(**cell)], temperature=10.0, neighbour_order=2, seed=seed)
    start = Start.tiled_grid(model, 8, 6, 6, 1)
    if types == 2:
        start.set_cell_types(1 + np.arange(start.n_cells) % 2)
    return start


def _replay(start, steps):
    replay = ReplayOracle.from_start(start)
    replay.step(steps)
    return replay


@pytest.mark.parametrize("kernel", sorted(KERNELS))
@pytest.mark.parametrize("term", ["volume", "surface"])
@pytest.mark.parametrize("target", [math.inf, -math.inf, math.nan, 3e38, 1e300])
@pytest.mark.parametrize("types", [1, 2])
def test_a_target_without_a_weight_changes_nothing(device, types, target, term, kernel, monkeypatch):
    for name, value in KERNELS[kernel].items():
        monkeypatch.setenv(f"GLAZIER_SWEEP_{name}", value)
    start = _start(types, target, term, weighted=False)
    replay = _replay(start, 8)
    assert replay.accepted > 100
    with device.GpuSimulation.from_start(start) as gpu:
        assert gpu.sweep_kernel == kernel
        gpu.step(8)
        assert np.array_equal(gpu.labels(), replay.labels())
        assert np.array_equal(gpu.volumes(), replay.volumes())
        assert np.array_equal(gpu.surfaces(), replay.surfaces())


@pytest.mark.parametrize("kernel", sorted(KERNELS))
@pytest.mark.parametrize("term", ["volume", "surface"])
@pytest.mark.parametrize("types", [1, 2])
def test_the_medium_has_no_target(device, types, term, kernel, monkeypatch):
    for name, value in KERNELS[kernel].items():
        monkeypatch.setenv(f"GLAZIER_SWEEP_{name}", value)
    start = _start(types, math.inf, term, weighted=True)
    replay = _replay(start, 8)
    with device.GpuSimulation.from_start(start) as gpu:
        assert gpu.sweep_kernel == kernel
        gpu.step(8)
        assert np.array_equal(gpu.labels(), replay.labels())
        assert np.array_equal(gpu.volumes(), replay.volumes())
        assert np.array_equal(gpu.surfaces(), replay.surfaces())


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("types", [1, 2])
def test_the_ensemble_prices_them_the_same(device, types, weighted):
    from glazier_b200.ensemble import Ensemble

    targets = [math.inf, 3e38] if weighted else [math.inf, math.nan, 3e38, 1e300]
    starts = [_start(types, target, term, weighted, seed=20 + i)
              for i, target in enumerate(targets) for term in ("volume", "surface")]
    want = [_replay(start, 8).labels() for start in starts]
    # the schedule it starts on, then the windowed kernel and blocks of 32 x 8
    for schedule in (None, 0, 2):
        ens = Ensemble(starts)
        if schedule is not None:
            ens.set_schedule(schedule)
        ens.step(8)
        for i in range(len(starts)):
            assert np.array_equal(ens.labels(i), want[i]), f"replica {i}"
        ens.close()
