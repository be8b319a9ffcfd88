"""The adjoint's tile kernels at the edges of tiles, launches and rounds.

Lattices smaller than a tile, of odd heights and with a last tile of a few
sites; rows that are not whole quads; up to four sub-steps a step (a launch takes four rounds) and five (the
one-round kernels); steps and checkpoint intervals that do not divide a
launch's steps; one to three species; 16 owner types (the most the tile
kernels hold) and 17.

The oracle is a plain f64 stencil under PyTorch autograd: fields within 1e-5
and gradients within 1e-4 of their largest value, the bounds the adjoint is
held to elsewhere. Fields and gradients are the same bits for every
checkpoint interval.
"""

from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MEDIUM = 255


def _plain(params, fields0, owners, w, h, ns, nt):
    import torch

    sec = params[2 * ns:2 * ns + nt * ns].reshape(nt, ns)
    upt = params[2 * ns + nt * ns:].reshape(nt, ns)
    u = [fields0[s].reshape(h, w) for s in range(ns)]
    for own in owners:
        own = own.reshape(h, w).long()
        cell = own != MEDIUM
        t = torch.where(cell, own, torch.zeros_like(own))
        for s in range(ns):
            k = max(1, math.ceil(float(params[s].detach()) / 0.25))
            v = u[s]
            for _ in range(k):
                faces = torch.roll(v, 1, 0) + torch.roll(v, -1, 0) + torch.roll(v, 1, 1) + torch.roll(v, -1, 1)
                v = v + params[s] / k * (faces - 4.0 * v) - params[ns + s] / k * v
            x = v + sec[:, s][t]
            x = (x - upt[:, s][t] * x).clamp(min=0.0)
            u[s] = torch.where(cell, x, v)
    return torch.stack(u).reshape(ns, h * w)


@pytest.mark.parametrize("w, h, diffusion, nt, steps", [
    (8, 6, (0.1,), 3, 9),
    (64, 32, (0.1, 0.2), 4, 8),
    (68, 33, (0.2, 0.05), 4, 11),
    (200, 97, (0.4, 0.1), 4, 7),
    (132, 70, (1.0, 0.1), 4, 6),
    (72, 40, (1.2, 0.2), 4, 5),
    (72, 65, (0.1, 0.3, 0.7), 16, 6),
    (72, 65, (0.1, 0.3, 0.7), 17, 6),
    # rows that are not whole quads: less than a region wide, a last tile of
    # one to three sites, a quad of the margin across the row's end
    (7, 6, (0.1,), 3, 9),
    (7, 6, (0.1, 0.2), 3, 9),
    (9, 7, (0.1, 0.6), 3, 9),
    (62, 33, (0.1, 0.2), 4, 8),
    (65, 32, (0.2, 0.05), 4, 11),
    (66, 40, (1.0, 0.1), 4, 6),
    (131, 70, (0.4, 0.1), 4, 7),
    (198, 97, (0.1, 0.3, 0.7), 16, 6),
    (258, 256, (0.1,), 3, 3),
])
def test_the_tiles_match_a_plain_stencil(device, w, h, diffusion, nt, steps):
    import torch

    from glazier_b200.adjoint import FieldAdjoint

    rng = np.random.default_rng(w * 1000 + h + nt)
    ns = len(diffusion)
    kinds = np.append(np.arange(1, nt), MEDIUM).astype(np.uint8)
    owners = np.stack([rng.choice(kinds, size=(h + 3) // 4 * ((w + 3) // 4)).reshape((h + 3) // 4, -1)
                       .repeat(4, 0).repeat(4, 1)[:h, :w].reshape(-1) for _ in range(steps)])
    params = np.concatenate([diffusion, rng.uniform(0.001, 0.02, ns), rng.uniform(0.0, 0.5, nt * ns),
                             rng.uniform(0.0, 0.1, nt * ns)])
    fields0 = rng.random((ns, h * w), dtype=np.float32)
    weight = rng.standard_normal((ns, h * w)).astype(np.float32)

    p = torch.from_numpy(params).requires_grad_()
    f = torch.from_numpy(fields0).double().requires_grad_()
    want = _plain(p, f, [torch.from_numpy(o) for o in owners], w, h, ns, nt)
    (want * torch.from_numpy(weight).double()).sum().backward()

    first = None
    for every in (1, 3, 4, steps):
        adj = FieldAdjoint(w, h, 1, ns, nt, owners, checkpoint_every=every)
        out = adj.forward(params, torch.from_numpy(fields0).cuda())
        gp, gf = adj.backward(torch.from_numpy(weight).cuda())
        adj.close()
        got = out.cpu().numpy(), gp, gf.cpu().numpy()
        if first is None:
            first = got
            for value, exact in zip(got, (want.detach().numpy(), p.grad.numpy(), f.grad.numpy())):
                bound = 1e-5 if value is got[0] else 1e-4
                assert np.abs(value - exact).max() <= bound * np.abs(exact).max()
        else:
            assert all(np.array_equal(a, b) for a, b in zip(got, first)), f"interval {every}"
