"""The direct sweep's forms at the edges of their ranges, against the replay.

- The two-field infection model (every term but motility) either side of each
  size from which its passes take another form, and a volume of every term
  past the size from which the gathering blocks are the wide ones: the default
  choices.
- Models of 16 and of 17 types, the most whose tables are held in shared
  memory and the least whose are read where they lie, with and without the
  terms past contact, volume and surface.
- The lean models' default choice either side of each of its sizes: the
  cluster up to (not with) 256^2 sites, in place up to one wave of blocks,
  gathered up to one wave of those, then streamed by warps; planes of few rows, whose cluster has CTAs without rows or a
  CTA that is its own neighbour; and a plane whose cluster threads take four
  targets each.

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


@pytest.mark.parametrize("size, kernel", [(512, "direct"), (514, "gathered"), (778, "gathered"), (780, "gathered"),
                                          (2046, "gathered"), (2048, "compact")])
def test_the_infection_model_either_side_of_each_size(device, size, kernel):
    """At 780^2 a pass has more targets than one wave of blocks, and the
    gathering blocks are the wide ones; from 2048^2 warps queue their own."""
    start = infection_start(seed=3, size=size, grid=size // 16, immune=64)
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
@pytest.mark.parametrize("kinds, width", [(16, 70), (17, 70), (16, 72), (17, 72)])
def test_tables_in_shared_memory_and_past_it(device, kinds, width, every, monkeypatch):
    """`kinds` types in all, on rows that are and are not whole multiples of
    four sites (the field step's two kernels); without the other terms the passes are launched
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
    model = Model(width=width, height=62, contact=contact, types=types, temperature=11.0, neighbour_order=2, seed=9)
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


@pytest.mark.parametrize("w, h, d, kernel", [
    (30, 2, 1, "cluster"), (18, 4, 1, "cluster"), (66, 34, 1, "cluster"), (130, 50, 1, "cluster"),
    (254, 256, 1, "cluster"), (256, 256, 1, "direct"), (778, 778, 1, "direct"), (780, 780, 1, "gathered"),
    (1100, 1102, 1, "gathered"), (1102, 1102, 1, "compact"), (2048, 2046, 1, "compact"), (2050, 2048, 1, "lean"),
    (80, 80, 80, "direct"), (88, 88, 88, "gathered"),
])
@pytest.mark.parametrize("types", [1, 2])
def test_the_lean_choice_either_side_of_each_size(device, w, h, d, kernel, types):
    side = 8 if min(w, h) >= 16 else 2
    gpu, replay = _lean(device, w, h, d, types, side)
    assert gpu.sweep_kernel == kernel
    _same(gpu, replay, 0)
    gpu.close()


@pytest.mark.parametrize("types", [1, 2])
def test_a_cluster_of_four_targets_a_thread(device, types, monkeypatch):
    monkeypatch.setenv("GLAZIER_SWEEP_RESIDENT", "1")
    gpu, replay = _lean(device, 512, 260, 1, types, 8)
    assert gpu.sweep_kernel == "cluster"
    _same(gpu, replay, 0)
    gpu.close()


def _lean(device, w, h, d, types, side):
    """The lean model of one or two types after 1 and then 4 MCS on both sides."""
    vt = float(side**2 if d == 1 else side**3)
    cell = dict(target_volume=vt, lambda_volume=1.0, target_surface=90.0, lambda_surface=0.05)
    model = Model(width=w, height=h, depth=d, contact=[0.0, 16.0, 16.0, 16.0, 6.0, 10.25, 16.0, 10.25, 9.125],
                  types=[CellType(), CellType(**cell), CellType(**cell)], temperature=10.0, neighbour_order=2, seed=5)
    start = Start.tiled(model, side)
    if types == 2:
        start.set_cell_types(1 + np.arange(start.n_cells) % 2)
    gpu = device.GpuSimulation.from_start(start)
    replay = ReplayOracle.from_start(start)
    for chunk in (1, 4):
        gpu.step(chunk)
        replay.step(chunk)
    return gpu, replay


@pytest.mark.parametrize("depth", [1, 16])
def test_many_divisions_and_deaths_in_a_step(device, depth):
    """Thousands of cells, most of which divide within a few steps, so a
    step's daughters are numbered over several chunks of labels, the label
    capacity grows during a call, and cells straddle the periodic edge."""
    w, h = (512, 500) if depth == 1 else (128, 100)
    side = 8 if depth == 1 else 4
    v = float(side**2 if depth == 1 else side**3)
    model = Model(width=w, height=h, depth=depth, contact=[0.0, 12.0, 12.0, 12.0, 8.0, 10.0, 12.0, 10.0, 8.0],
                  types=[CellType(), CellType(target_volume=2 * v, lambda_volume=2.0, division_volume=1.05 * v),
                         CellType(target_volume=v, lambda_volume=2.0, death_rate=0.02)],
                  temperature=12.0, neighbour_order=2, seed=13)
    start = Start.tiled(model, side)
    start.set_cell_types(1 + (np.arange(start.n_cells) % 7 == 3))
    gpu = device.GpuSimulation.from_start(start)
    replay = ReplayOracle.from_start(start)
    for chunk in (3, 17):
        gpu.step(chunk)
        replay.step(chunk)
        assert gpu.n_labels == replay.n_labels
        _same(gpu, replay, 0)
    # more labels than one chunk of the decision holds, and divisions among them
    assert start.n_cells > 2048 and gpu.n_labels > start.n_cells + 1
    gpu.close()


def test_a_volume_of_every_term_in_wide_blocks(device):
    """More than 148 x 4 x 256 targets a pass, with the veto, motility, drift,
    chemotaxis, length, death and a field of two sub-steps."""
    cell = dict(target_volume=216.0, lambda_volume=2.0, connected=True, max_activity=20.0, lambda_activity=60.0,
                external=(0.0, 0.0, 1.0), death_rate=0.002, target_surface=300.0, lambda_surface=0.05)
    model = Model(width=108, height=110, depth=104, contact=[0.0, 16.0, 16.0, 16.0, 8.0, 9.0, 16.0, 9.0, 8.0],
                  types=[CellType(), CellType(**cell), CellType(target_length=8.0, lambda_length=0.5, **cell)],
                  temperature=10.0, neighbour_order=2, seed=29, species=[Species("signal", 0.3, 0.01, 0.0)],
                  secretion=[[0.0], [0.2], [0.1]], uptake=[[0.0], [0.0], [0.05]], chemotaxis=[[0.0], [10.0], [5.0]])
    start = Start.tiled(model, 6)
    start.set_cell_types(1 + np.arange(start.n_cells) % 2)
    gpu = device.GpuSimulation.from_start(start)
    assert gpu.sweep_kernel == "gathered" and model.sites // 8 > 148 * 4 * 256
    replay = ReplayOracle.from_start(start)
    gpu.step(3)
    replay.step(3)
    _same(gpu, replay, 1)
    gpu.close()


@pytest.mark.parametrize("depth", [1, 12])
@pytest.mark.parametrize("top", [20.0, 20.5, 255.0, 256.0, 300.0])
def test_activities_in_the_log_table_and_past_it(device, depth, top):
    """Act memories that run through whole activities below 256 (read from a
    block's table of logs), through halves, and past the table."""
    cell = dict(target_volume=64.0, lambda_volume=2.0, max_activity=top, lambda_activity=80.0)
    model = Model(width=48, height=44, depth=depth, contact=[0.0, 16.0, 16.0, 16.0, 8.0, 9.0, 16.0, 9.0, 8.0],
                  types=[CellType(), CellType(**cell), CellType(target_volume=64.0, lambda_volume=2.0)],
                  temperature=12.0, neighbour_order=2, seed=31)
    start = Start.tiled(model, 8 if depth == 1 else 4)
    start.set_cell_types(1 + np.arange(start.n_cells) % 2)
    gpu = device.GpuSimulation.from_start(start)
    replay = ReplayOracle.from_start(start)
    gpu.step(15)
    replay.step(15)
    _same(gpu, replay, 0)
    gpu.close()


def test_deaths_without_divisions_keep_no_moments(device):
    """Death alone needs no moment sums: every form of the pass still follows
    the replay through the deaths."""
    model = Model(width=96, height=80, contact=[0.0, 16.0, 16.0, 8.0],
                  types=[CellType(), CellType(target_volume=64.0, lambda_volume=2.0, death_rate=0.05)],
                  temperature=10.0, neighbour_order=2, seed=37)
    start = Start.tiled(model, 8)
    gpu = device.GpuSimulation.from_start(start)
    replay = ReplayOracle.from_start(start)
    for chunk in (1, 9, 20):
        gpu.step(chunk)
        replay.step(chunk)
        _same(gpu, replay, 0)
    assert int((gpu.volumes()[1:] == 0).sum()) > 0
    gpu.close()


@pytest.mark.parametrize("w, h, d", [(32, 32, 1), (64, 66, 1), (126, 62, 1), (514, 70, 1), (18, 10, 6), (34, 30, 22)])
@pytest.mark.parametrize("ctas", ["1", "2"])
@pytest.mark.parametrize("types", [1, 2])
def test_warps_that_stream_over_runs(device, w, h, d, ctas, types, monkeypatch):
    """The lean models on one or two blocks' warps: runs of one whole step of
    128 targets and less, of a step and a part, of many steps that carry
    entries over, a last warp's short run and warps without a target."""
    monkeypatch.setenv("GLAZIER_SWEEP_DIRECT", "0")
    monkeypatch.setenv("GLAZIER_SWEEP_CTAS", ctas)
    gpu, replay = _lean(device, w, h, d, types, 8 if d == 1 else 2)
    assert gpu.sweep_kernel == "lean"
    _same(gpu, replay, 0)
    gpu.close()
