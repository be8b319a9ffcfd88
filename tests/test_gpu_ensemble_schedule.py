"""The schedule an ensemble starts on can be taken again by its number, and no
number past it is one."""

from __future__ import annotations

import numpy as np
import pytest

from glazier_b200.workloads import monolayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 24])
def test_the_first_schedule_has_a_number(device, depth):
    from glazier_b200.ensemble import Ensemble

    starts = [monolayer(size, depth=depth, seed=i) for i, size in enumerate((24, 40))]
    with Ensemble(starts) as ens, Ensemble(starts) as ref:
        ref.step(6)
        ens.step(2)
        ens.set_schedule(0)
        ens.step(2)
        ens.set_schedule(16)
        ens.step(2)
        for i in range(len(starts)):
            assert np.array_equal(ens.labels(i), ref.labels(i))
        for schedule in (-1, 17, 18, 24, 32):
            with pytest.raises(device.GpuError, match="no such schedule"):
                ens.set_schedule(schedule)
