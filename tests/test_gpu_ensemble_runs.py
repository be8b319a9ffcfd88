"""The batch's kernels in every form, against the replay.

The runs of consecutive targets that an ensemble starts on, and the windowed
kernel with its windows by tensor copies and by plain loads, in planes of four
and eight neighbours and in volumes of 6, 18 and 26; of one type whose contact
sum is a product, of one whose is not exact, of two types, and of 16 and 17
(the most whose tables are held in shared memory and the least whose are read
where they lie). Sides are uneven, and a replica's last run is a short one, or
its only one. Every replica's lattice, volumes and surfaces are the replay's,
bit for bit.
"""

from __future__ import annotations

import os

import numpy as np
import pytest

from glazier_b200.blueprint import CellType, Model, Start
from oracle.replay import ReplayOracle

pytestmark = pytest.mark.gpu

PLANES = [(64, 64, 1), (72, 62, 1), (124, 34, 1), (16, 10, 1)]
VOLUMES = [(24, 18, 14), (32, 34, 20), (68, 10, 12), (8, 4, 4)]


@pytest.fixture(autouse=True)
def _default_kernels(monkeypatch):
    for name in list(os.environ):
        if name.startswith("GLAZIER_"):
            monkeypatch.delenv(name)


def _start(shape, order: int, types: int, exact: bool, seed: int) -> Start:
    w, h, d = shape
    side = 4
    v = float(side**2 if d == 1 else side**3)
    n = types + 1
    contact = [0.0 if a == b == 0 else 6.0 + (a * 5 + b * 5 + a * b) % 7 + (0.0 if exact else 0.1)
               for a in range(n) for b in range(n)]
    cells = [CellType(target_volume=v + t, lambda_volume=1.0 + 0.25 * (t % 3), target_surface=30.0 + t,
                      lambda_surface=0.05 * (t % 2)) for t in range(1, n)]
    model = Model(width=w, height=h, depth=d, contact=contact, types=[CellType(), *cells], temperature=9.0 + seed % 3,
                  neighbour_order=order, seed=seed)
    start = Start.tiled(model, side)
    start.set_cell_types(1 + np.arange(start.n_cells) % types)
    return start


# (the ensemble's schedule, None the one it starts on; tensor copies)
@pytest.mark.parametrize("schedule, tma", [(None, "1"), (0, "1"), (0, "0")])
@pytest.mark.parametrize("types, exact", [(1, True), (1, False), (2, True), (15, True), (16, True)])
@pytest.mark.parametrize("order, volume", [(1, False), (2, False), (1, True), (2, True), (3, True)])
def test_every_form_reproduces_the_replay(device, order, volume, types, exact, schedule, tma, monkeypatch):
    from glazier_b200.ensemble import Ensemble

    monkeypatch.setenv("GLAZIER_SWEEP_TMA", tma)
    starts = [_start(shape, order, types, exact, seed=40 + i) for i, shape in enumerate(VOLUMES if volume else PLANES)]
    ens = Ensemble(starts)
    if schedule is not None:
        ens.set_schedule(schedule)
    ens.step(1)
    ens.step(6)
    for i, start in enumerate(starts):
        replay = ReplayOracle.from_start(start)
        replay.step(7)
        assert np.array_equal(ens.labels(i), replay.labels()), f"replica {i}"
        assert np.array_equal(ens.volumes(i), replay.volumes()), f"replica {i}"
        assert np.array_equal(ens.surfaces(i), replay.surfaces()), f"replica {i}"
    ens.close()
