"""Adjoint handles through a refused allocation, and beside one another."""

from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MEDIUM = 255


def _inputs(w, h, ns, nt, steps, seed):
    rng = np.random.default_rng(seed)
    kinds = np.append(np.arange(nt), MEDIUM).astype(np.uint8)
    owners = rng.choice(kinds, size=(steps, h * w))
    params = np.concatenate([np.full(ns, 0.1), np.full(ns, 0.01), rng.uniform(0.0, 0.5, nt * ns),
                             rng.uniform(0.0, 0.1, nt * ns)])
    fields = rng.random((ns, h * w), dtype=np.float32)
    weight = rng.standard_normal((ns, h * w)).astype(np.float32)
    return owners, params, fields, weight


def _gradients(adj, params, fields, weight):
    import torch

    out = adj.forward(params, torch.from_numpy(fields).cuda())
    gp, gf = adj.backward(torch.from_numpy(weight).cuda())
    return out.cpu().numpy(), gp, gf.cpu().numpy()


def test_a_refused_buffer_leaves_the_handle_usable(device):
    """Sub-step counts whose states no device holds are refused; the handle's
    next run takes new buffers and gives what it gave before."""
    from glazier_b200.adjoint import FieldAdjoint
    from glazier_b200.engine import GpuError

    w, h, ns, nt, steps = 72, 40, 2, 4, 6
    owners, params, fields, weight = _inputs(w, h, ns, nt, steps, 3)
    adj = FieldAdjoint(w, h, 1, ns, nt, owners, checkpoint_every=3)
    want = _gradients(adj, params, fields, weight)
    # 2e8 sub-steps a step: 3 * 2e8 * 2 * 2880 floats
    more = params.copy()
    more[0] = 5e7
    with pytest.raises(GpuError, match="out of memory"):
        _gradients(adj, more, fields, weight)
    other = FieldAdjoint(w, h, 1, ns, nt, owners, checkpoint_every=2)  # may take the freed memory
    alone = _gradients(other, params, fields, weight)
    for _ in range(2):
        got = _gradients(adj, params, fields, weight)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert all(np.array_equal(a, b) for a, b in zip(_gradients(other, params, fields, weight), alone))
    adj.close()
    other.close()


# (width, height, species, types): the tile kernels at one, four and 16 types,
# the round kernels at 17, at 40, and on a row that is not whole quads
SHAPES = [(64, 40, 2, 1), (64, 40, 2, 16), (72, 33, 1, 4), (64, 40, 2, 17), (64, 40, 2, 40), (66, 20, 1, 60)]


def test_handles_of_different_types_side_by_side(device):
    from glazier_b200.adjoint import FieldAdjoint

    steps = 6
    inputs = [_inputs(*shape, steps, seed) for seed, shape in enumerate(SHAPES)]

    def make(i):
        w, h, ns, nt = SHAPES[i]
        return FieldAdjoint(w, h, 1, ns, nt, inputs[i][0], checkpoint_every=3)

    want = []
    for i in range(len(SHAPES)):
        adj = make(i)
        want.append(_gradients(adj, *inputs[i][1:]))
        adj.close()

    # alive together: graphs captured while the others' kernels were set up
    handles = [make(i) for i in range(len(SHAPES))]
    for _ in range(2):
        for i, adj in enumerate(handles):
            got = _gradients(adj, *inputs[i][1:])
            assert all(np.array_equal(a, b) for a, b in zip(got, want[i])), f"handle {i}"
    for adj in handles:
        adj.close()

    wrong = []

    def drive(i):
        try:
            for _ in range(30):
                adj = make(i)
                got = _gradients(adj, *inputs[i][1:])
                adj.close()
                if not all(np.array_equal(a, b) for a, b in zip(got, want[i])):
                    wrong.append(f"handle {i}")
        except Exception as exc:  # reported on the main thread
            wrong.append(f"handle {i}: {exc}")

    threads = [threading.Thread(target=drive, args=(i,)) for i in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
