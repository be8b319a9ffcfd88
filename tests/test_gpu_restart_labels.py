"""A restart from a lattice with labels past the label count.

Such sites become medium before any sweep reads them, and the next step still
fails with the status that names them. The run is the replay's from the
lattice with those sites medium, bit for bit, whichever kernel takes it.
"""

from __future__ import annotations

import os

import numpy as np
import pytest

from conftest import sheet_model, tiled
from glazier_b200.blueprint import Start
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu

PLANE = dict(width=96, height=64)
MODELS = {
    "cluster": dict(PLANE),
    "direct": dict(PLANE, target_length=12.0, lambda_length=1.0),
    "population": dict(PLANE, division_volume=80.0, death_rate=0.01),
    "volume": dict(width=24, height=20, depth=18, order=3, target_volume=512.0),
}


@pytest.fixture(autouse=True)
def _default_kernels(monkeypatch):
    for name in list(os.environ):
        if name.startswith("GLAZIER_"):
            monkeypatch.delenv(name)


@pytest.mark.parametrize("device_input", [False, True])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_sites_past_the_label_count_become_medium(device, name, device_input):
    start = tiled(sheet_model(seed=7, **MODELS[name]))
    n, sites = start.cell_type.size, start.model.sites
    rng = np.random.default_rng(5)
    bad = np.unique(np.concatenate([[0, 1, sites - 1], rng.integers(0, sites, 200)]))
    labels = start.labels.copy()
    labels[bad] = np.resize(np.array([n, n + 1, 2**31 - 1, 2**31, 2**32 - 1], dtype=np.uint32), bad.size)
    clean = start.labels.copy()
    clean[bad] = 0
    sim = device.GpuSimulation.from_start(start)
    if device_input:
        import torch

        sim.set_labels_tensor(torch.from_numpy(labels.view(np.int32)).cuda())
    else:
        sim.set_labels(labels)
    assert np.array_equal(sim.labels(), clean)
    with pytest.raises(device.GpuError, match="not below the cell type count"):
        sim.step(3)
    replay = ReplayOracle.from_start(Start(start.model, clean, start.cell_type))
    replay.step(3)
    assert np.array_equal(sim.labels(), replay.labels())
    assert sim.n_labels == replay.n_labels
    assert np.array_equal(sim.volumes(), replay.volumes())
    assert np.array_equal(sim.surfaces(), replay.surfaces())
    sim.close()
