"""The calls whose speed this framework is judged by, one dict of plain values each.

`listed()` names the fixed cases, `draw(rng)` makes one more from the same
ranges, `prepare(case, seed)` builds what a user's program holds before the
call, `run(state)` is one pass through the public entry points, `work(case)`
the least bytes and operations of that pass and `exact(case, seed)` the same
outputs in 64 bits where a plain computation gives them.

Kinds of case:

- "sweep"     an engine of contact, volume and surface terms kept between
              calls and stepped: `GpuSimulation.step`, then the lattice read in
              place (`labels_tensor`). What a monolayer, sorting or volume
              study does, and, with one MCS a call, what a loop that couples
              another solver to the lattice does.
- "tissue"    the same with the other terms on: two diffusing fields,
              chemotaxis, a length constraint, several types.
- "job"       a whole run as `glazier_b200.native.run` or the command-line
              runner makes it: engine from a start, every MCS, the lattice,
              cells and fields read back. Models with division, death,
              infection, connectivity and motility, whose state does not come
              back to where it was, are measured as whole runs.
- "ensemble"  many replicas of uneven sizes stepped as one, every lattice read.
- "adjoint"   one training step through the differentiable field step: forward,
              loss, backward, gradients.
"""

from __future__ import annotations

import json
import math

import numpy as np
import torch

from glazier_b200 import workloads
from glazier_b200.adjoint import MEDIUM, FieldAdjoint, field_trajectory
from glazier_b200.blueprint import Blueprint, CellType, Model, Start
from glazier_b200.engine import GpuSimulation
from glazier_b200.ensemble import Ensemble


def listed() -> list:
    return [
        # one MCS a call on the plain monolayer: a coupling loop that looks at
        # the lattice after every step; launches and host latency are all there is
        dict(name="coupled-step-128", kind="sweep", w=128, h=128, d=1, mcs=1, types=1, surface=False, order=2),
        # the plain monolayer at its published size, 100 MCS a call
        dict(name="monolayer-128", kind="sweep", w=128, h=128, d=1, mcs=100, types=1, surface=False, order=2),
        # cell sorting: two types of different adhesion
        dict(name="sorting-512", kind="sweep", w=512, h=512, d=1, mcs=100, types=2, surface=False, order=2),
        # the scaling sweep of the monolayer with its surface term
        dict(name="monolayer-1024", kind="sweep", w=1024, h=1024, d=1, mcs=50, types=1, surface=True, order=2),
        dict(name="monolayer-4096", kind="sweep", w=4096, h=4096, d=1, mcs=10, types=1, surface=True, order=2),
        # the scaling sweep's volume, 26 neighbours
        dict(name="volume-128", kind="sweep", w=128, h=128, d=128, mcs=20, types=1, surface=True, order=3),
        # two fields, chemotaxis and length terms on a plane
        dict(name="tissue-512", kind="tissue", w=512, mcs=50),
        # the same past the sizes that are priced without staging
        dict(name="tissue-2048", kind="tissue", w=2048, mcs=10),
        # the two-field infection model, whole: division, death, infection,
        # connectivity, chemotaxis, length, 200 MCS
        dict(name="infection-256-job", kind="job", model="infection", w=256, mcs=200),
        # an infected slab with motile immune cells, whole: 18 neighbours, the
        # veto over the 26 ring, a field of three sub-steps, death
        dict(name="slab-64x64x32-job", kind="job", model="slab", w=64, d=32, mcs=60),
        # 64 replicas of uneven sizes and parameters, 100 MCS a call
        dict(name="ensemble-64", kind="ensemble", count=64, low=128, high=1024, shapes=1, mcs=100),
        # the field adjoint: 50 steps, a checkpoint every 10
        dict(name="adjoint-512", kind="adjoint", w=512, h=512, species=2, steps=50, every=10, fast=False),
    ]


def _even(rng, low: float, high: float) -> int:
    """An even side, log-uniform from `low` to `high`."""
    return 2 * max(1, round(math.exp(rng.uniform(math.log(low), math.log(high))) / 2))


def draw(rng) -> dict:
    kind = rng.choice(["plane", "plane", "plane", "volume", "volume", "tissue", "job", "slab", "ensemble", "adjoint"])
    if kind == "plane":
        w, h = _even(rng, 64, 4096), _even(rng, 64, 4096)
        most = max(1, int(1.6e8 / (w * h)))
        mcs = min(rng.choice([1, 5, 20, 100]), most)
        return dict(kind="sweep", w=w, h=h, d=1, mcs=mcs, types=rng.choice([1, 1, 2]), surface=rng.random() < 0.5,
                    order=rng.choice([1, 2, 2, 2]))
    if kind == "volume":
        w, h, d = (_even(rng, 24, 192) for _ in range(3))
        most = max(1, int(6e7 / (w * h * d)))
        return dict(kind="sweep", w=w, h=h, d=d, mcs=min(rng.choice([1, 5, 20]), most), types=rng.choice([1, 1, 2]),
                    surface=rng.random() < 0.5, order=rng.choice([1, 2, 3, 3]))
    if kind == "tissue":
        w = 8 * max(8, round(math.exp(rng.uniform(math.log(96), math.log(2048))) / 8))
        return dict(kind="tissue", w=w, mcs=max(2, min(50, int(4e7 / (w * w)))))
    if kind == "job":
        return dict(kind="job", model="infection", w=_even(rng, 128, 512), mcs=rng.randint(50, 200))
    if kind == "slab":
        return dict(kind="job", model="slab", w=8 * rng.randint(3, 10), d=8 * rng.randint(2, 5),
                    mcs=rng.randint(10, 60))
    if kind == "ensemble":
        low = rng.choice([64, 128])
        return dict(kind="ensemble", count=rng.randint(8, 48), low=low, high=low * rng.choice([2, 4, 8]),
                    shapes=rng.randint(1, 1000), mcs=rng.randint(10, 100))
    w, h = _even(rng, 96, 1024), _even(rng, 96, 1024)
    steps = rng.randint(10, 60)
    return dict(kind="adjoint", w=w, h=h, species=rng.choice([1, 2, 2]), steps=steps,
                every=min(steps, rng.choice([5, 10, 20])), fast=rng.random() < 0.25)


# ------------------------------------------------------------------ starts


def _sweep_start(case: dict, seed: int) -> Start:
    """A lattice tiled by cells of side 8: the plain monolayer (or volume), or
    two types whose adhesion sorts them (the contact energies and fractions
    of the molecular-adhesion monolayer)."""
    w, h, d = case["w"], case["h"], case["d"]
    side = 8
    vt = float(side**2 if d == 1 else side**3)
    surface = dict(lambda_surface=0.2, target_surface=workloads.initial_surface(side, d)) if case["surface"] else {}
    if case["types"] == 1:
        contact, types = [0.0, 10.0, 10.0, 10.0], [CellType(), CellType(target_volume=vt, lambda_volume=1.0, **surface)]
    else:
        contact = [0.0, 16.0, 16.0, 16.0, 6.0, 10.25, 16.0, 10.25, 9.125]
        cell = CellType(target_volume=vt, lambda_volume=2.0, **surface)
        types = [CellType(), cell, cell]
    model = Model(width=w, height=h, depth=d, contact=contact, types=types, temperature=10.0,
                  neighbour_order=case["order"], seed=1 + seed)
    start = Start.tiled(model, side)
    if case["types"] == 2:
        kinds = 1 + (np.random.default_rng(seed).random(start.n_cells) < 0.25)
        start.set_cell_types(kinds.astype(np.uint8))
    return start


_SLAB = {
    "name": "an infected slab with motile immune cells",
    "types": [
        {"name": "Epithelial", "target_volume": 512.0, "lambda_volume": 2.0, "target_surface": 320.0,
         "lambda_surface": 0.05, "connected": True, "secretion": {"virus": 0.02}, "death_rate": 0.001},
        {"name": "Immune", "target_volume": 512.0, "lambda_volume": 2.0, "max_activity": 100.0,
         "lambda_activity": 100.0, "uptake": {"virus": 0.05}, "chemotaxis": {"virus": 150.0}},
    ],
    "fields": [{"name": "virus", "diffusion": 0.5, "decay": 0.01, "initial": 0.0}],
    "contact": [0.0, 16.0, 16.0, 16.0, 8.0, 12.0, 16.0, 12.0, 10.0],
    "temperature": 10.0,
    "neighbour_order": 2,
    "dump_every": 0,
    "units": {"micron_per_site": 1.0, "minute_per_step": 1.0},
}


def _slab_start(case: dict, seed: int) -> Start:
    w, d = case["w"], case["d"]
    text = dict(_SLAB, width=w, height=w, depth=d, seed=3 + seed, steps=case["mcs"],
                initial={"side": 8, "nx": w // 8, "ny": w // 8, "nz": d // 8, "fractions": {"Immune": 0.08}})
    return Blueprint.from_json(json.dumps(text)).start()


# ----------------------------------------------------------------- adjoint

_SECRETION = [[0.0, 0.0], [0.0, 0.0], [1.0, 0.5], [0.0, 0.0]]  # [type][species]: medium, healthy, infected, immune
_UPTAKE = [[0.0, 0.0], [0.02, 0.0], [0.0, 0.0], [0.0, 0.01]]


def _adjoint_inputs(case: dict, seed: int):
    """Parameters (D, decay per species; secretion, uptake per type and
    species), initial fields, an owner trajectory and observed fields.

    The trajectory is a tiling of cells of side 8, one in 16 infected and a
    few immune, whose borders move by copies of random neighbours, as the
    sweep moves them; the observed fields come from parameters up to 10 % off.
    """
    w, h, ns, steps = case["w"], case["h"], case["species"], case["steps"]
    rng = np.random.default_rng(seed)
    cells = np.add.outer(np.arange(h) // 8 * (-(-w // 8)), np.arange(w) // 8)
    kind = rng.choice(np.array([1, 2, 3, MEDIUM], dtype=np.uint8), size=cells.max() + 1, p=[0.88, 0.06, 0.02, 0.04])
    trajectory = np.empty((steps, h * w), dtype=np.uint8)
    for t in range(steps):
        axis, shift = (0, 1)[t & 1], (1, -1)[(t >> 1) & 1]
        cells = np.where(rng.random((h, w), dtype=np.float32) < 0.08, np.roll(cells, shift, axis), cells)
        trajectory[t] = kind[cells].reshape(-1)
    diffusion = np.array([0.4, 0.8] if case["fast"] else [0.05, 0.1])[:ns]
    params = np.concatenate([diffusion, np.array([0.01, 0.005])[:ns], np.array(_SECRETION)[:, :ns].reshape(-1),
                             np.array(_UPTAKE)[:, :ns].reshape(-1)])
    fields0 = rng.random((ns, h * w), dtype=np.float32)
    off = params * (1.0 + 0.1 * (2.0 * rng.random(params.size) - 1.0))
    fields0 = torch.from_numpy(fields0).cuda()
    owners = torch.from_numpy(trajectory).cuda()
    with torch.no_grad():
        observed = _plain_fields(case, torch.from_numpy(off).cuda(), fields0.double(), owners).float()
    return params, fields0, trajectory, owners, observed


def _plain_fields(case: dict, params, fields0, owners):
    """The field step over the trajectory in plain torch: k sub-steps of
    diffusion and decay, then secretion and uptake by the owner of each site."""
    w, h, ns = case["w"], case["h"], case["species"]
    nt = 4
    sec = params[2 * ns: 2 * ns + nt * ns].reshape(nt, ns)
    upt = params[2 * ns + nt * ns:].reshape(nt, ns)
    u = [fields0[s].reshape(h, w) for s in range(ns)]
    for t in range(case["steps"]):
        own = owners[t].reshape(h, w).long()
        cell = own != MEDIUM
        own = torch.where(cell, own, torch.zeros_like(own))
        for s in range(ns):
            k = max(1, math.ceil(float(params[s].detach()) / 0.25))
            v = u[s]
            for _ in range(k):
                faces = torch.roll(v, 1, 0) + torch.roll(v, -1, 0) + torch.roll(v, 1, 1) + torch.roll(v, -1, 1)
                v = v + params[s] / k * (faces - 4.0 * v) - params[ns + s] / k * v
            x = v + sec[:, s][own]
            x = (x - upt[:, s][own] * x).clamp(min=0.0)
            u[s] = torch.where(cell, x, v)
    return torch.stack(u).reshape(ns, h * w)


# --------------------------------------------------------- prepare and run


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "sweep":
        return dict(case=case, sim=GpuSimulation.from_start(_sweep_start(case, seed)))
    if kind == "tissue":
        return dict(case=case, sim=GpuSimulation.from_start(workloads.adjoint_start(seed=1 + seed, size=case["w"])))
    if kind == "job":
        if case["model"] == "slab":
            return dict(case=case, start=_slab_start(case, seed), rule=None)
        w = case["w"]
        start = workloads.infection_start(seed=1 + seed, size=w, grid=w // 16, immune=w * w // 2048)
        return dict(case=case, start=start, rule=workloads.INFECTION_RULE)
    if kind == "ensemble":
        # the sides and parameters are the case's; the replicas' own random draws follow the seed
        starts = workloads.ensemble_starts(case["count"], seed=case["shapes"], low=case["low"], high=case["high"])
        for i, start in enumerate(starts):
            start.model.seed = seed * 4096 + i
        ens = Ensemble(starts)
        ens.autotune(3)
        return dict(case=case, ens=ens)
    params, fields0, trajectory, _, observed = _adjoint_inputs(case, seed)
    adj = FieldAdjoint(case["w"], case["h"], 1, case["species"], 4, trajectory, checkpoint_every=case["every"])
    return dict(case=case, adj=adj, params=torch.from_numpy(params), fields0=fields0, observed=observed)


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "sweep":
        state["sim"].step(case["mcs"])
        return state["sim"].labels_tensor()
    if kind == "tissue":
        sim = state["sim"]
        sim.step(case["mcs"])
        return [sim.labels_tensor(), sim.field_tensor(0), sim.field_tensor(1)]
    if kind == "job":
        with GpuSimulation.from_start(state["start"]) as sim:
            if state["rule"] is not None:
                sim.set_infection(*state["rule"])
            sim.step(case["mcs"])
            species = len(state["start"].model.species)
            return [sim.labels(), sim.volumes(), sim.cell_types()] + [sim.field(s) for s in range(species)]
    if kind == "ensemble":
        state["ens"].step(case["mcs"])
        return [state["ens"].labels(i) for i in range(case["count"])]
    params = state["params"].detach().requires_grad_()
    fields0 = state["fields0"].detach().requires_grad_()
    out = field_trajectory(params, fields0, state["adj"])
    ((out - state["observed"]) ** 2).mean().backward()
    return [out.detach(), params.grad, fields0.grad]


def _sites(case: dict) -> int:
    kind = case["kind"]
    if kind == "sweep":
        return case["w"] * case["h"] * case["d"]
    if kind == "ensemble":
        # the replicas' mean area: sides log-uniform from low to high
        ratio = case["high"] / case["low"]
        mean = case["low"] ** 2 * (ratio**2 - 1.0) / (2.0 * math.log(ratio))
        return int(case["count"] * mean)
    if kind == "adjoint":
        return case["w"] * case["h"]
    return case["w"] ** 2 * case.get("d", 1)


def work(case: dict) -> dict:
    """A Monte Carlo step reads every label once and writes the lattice once,
    and each field once in and out; about a fifth of its copy attempts meet
    another label and price their neighbourhood. The adjoint reads the owners
    and the fields and writes the fields and gradients once."""
    kind, sites = case["kind"], _sites(case)
    if kind == "adjoint":
        ns, steps = case["species"], case["steps"]
        k = 4 if case["fast"] else 1
        return {"bytes": sites * (steps + 16.0 * ns), "flops": sites * steps * ns * (8.0 * k + 24.0 * k + 8.0)}
    if kind == "sweep":
        offsets = {1: 4, 2: 8, 3: 8}[case["order"]] if case["d"] == 1 else {1: 6, 2: 18, 3: 26}[case["order"]]
        species = 0
    else:
        offsets = 18 if case.get("model") == "slab" else 8
        species = 0 if kind == "ensemble" else (1 if case.get("model") == "slab" else 2)
    per_site = 8.0 + species * 8.0
    return {"bytes": case["mcs"] * sites * per_site,
            "flops": case["mcs"] * sites * (0.2 * (2.0 * offsets + 20.0) + species * 12.0)}


def exact(case: dict, seed: int):
    """The adjoint's fields and gradients in f64. A sweep's lattice, and the
    fields that follow it, come from the engine's own random draws and have no
    value apart from them."""
    if case["kind"] != "adjoint":
        return None
    params, fields0, _, owners, observed = _adjoint_inputs(case, seed)
    p = torch.from_numpy(params).cuda().requires_grad_()
    f = fields0.double().requires_grad_()
    out = _plain_fields(case, p, f, owners)
    ((out - observed.double()) ** 2).mean().backward()
    return [out.detach(), p.grad, f.grad]
