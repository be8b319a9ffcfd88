"""An error that a call has reported is not reported again by a later one."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import sheet_model, tiled

pytestmark = pytest.mark.gpu


def test_a_refused_allocation_is_not_the_next_launch_s_error(device):
    import torch

    from glazier_b200.adjoint import FieldAdjoint
    from glazier_b200.ensemble import Ensemble

    w = h = 64
    # 2e8 sub-steps a step: their states fit no device
    params = np.array([5e7, 0.01, 0.0, 0.1, 0.0, 0.02])
    adj = FieldAdjoint(w, h, 1, 1, 2, np.ones((2, w * h), dtype=np.uint8), checkpoint_every=1)
    fields = torch.zeros((1, w * h), device="cuda")

    def refuse():
        with pytest.raises(device.GpuError, match="out of memory"):
            adj.forward(params, fields)

    start = tiled(sheet_model(seed=3))
    refuse()
    sim = device.GpuSimulation.from_start(start)
    sim.step(2)
    refuse()
    assert sim.volumes().sum() == w * h
    refuse()
    sim.set_labels(start.labels)
    refuse()
    with Ensemble([start]) as ens:
        refuse()
        ens.step(2)
        assert ens.volumes(0).sum() == w * h
    sim.close()
    adj.close()
