"""What a user of this framework has it do, as cases that can be timed and
compared: whole contact-dynamics steps of colonies from a few hundred cells to
a million (host arrays and device-resident ones, open colonies and walled
traps, with and without flow drift and growth-load laws), batches of
independent colonies, and the contact search, wall contacts, contact graph,
contact solve and warm-start network through their own entry points.

Colonies are laid out by ``settled_colony``: capsules in aligned tracks, end
to end with small gaps and overlaps, as a jammed colony looks between two
steps of its growth (+1 % length a step, some pairs overlapping by what a step
or a division leaves).  ``workloads`` gives the two starts that are random on
purpose: the 1,000-capsule colony and the trap.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from microsimulator_b200 import abi, learned, workloads
from microsimulator_b200.backend import B200Backend, DeviceCells, DeviceOutputs
from microsimulator_b200.graph import device_index
from microsimulator_b200.simulation import Simulation
from microsimulator_b200.sweep import ColonyBatch
from microsimulator_b200.types import (
    ConstraintContactParameters,
    ContactDynamicsParameters,
    ContactParameters,
    ContactSolveParameters,
    ContactSystem,
    FlowField,
    GrowthLoadLaw,
    GrowthLoadResponse,
    empty_bodies,
    empty_rows,
)
from microsimulator_b200.world import WorldState, normalized_arrays

DT = 0.02
TOLERANCE = 5e-4  # um: 1e-3 capsule radii, the benchmark's
GROWTH = 0.5  # +1 % length a step
RADIUS = workloads.RADIUS
CONTACTS = 1.3  # contacts a cell of the contact lists and systems made here
GEOMETRY = ("position_x", "position_y", "position_z", "direction_x", "direction_y", "direction_z", "lengths")
LAWS = {
    "none": GrowthLoadResponse(),
    "linear": GrowthLoadResponse(GrowthLoadLaw.LINEAR, 0.0, 0.2, 3.0),
    "exponential": GrowthLoadResponse(GrowthLoadLaw.EXPONENTIAL, 0.4, 0.0, 1.0),
}


def listed():
    return [
        # An interactive program stepping a young colony held in host arrays:
        # launches and round trips are all there is.
        {"name": "step_host_300", "kind": "step", "cells": 300, "start": "settled", "resident": False, "law": "none"},
        # The first step of the 1,000-capsule colony from its random,
        # overlapping start: several substeps, thousands of iterations.
        {"name": "start_1k", "kind": "step", "cells": 1000, "start": "random", "resident": False, "law": "none"},
        # A colony between the two, device-resident, with load-limited growth.
        {"name": "step_20k_load", "kind": "step", "cells": 20011, "start": "settled", "resident": True,
         "law": "linear"},
        # A colony drifting in a channel's flow.
        {"name": "step_60k_flow", "kind": "step", "cells": 60000, "start": "flow", "resident": True, "law": "none"},
        # The trap with its four wall boxes.
        {"name": "trap_100k", "kind": "step", "cells": 100000, "start": "trap", "resident": True, "law": "none"},
        # The benchmark's size.
        {"name": "step_1m", "kind": "step", "cells": 1000000, "start": "settled", "resident": True, "law": "none"},
        # A parameter sweep: independent colonies stepped by one call.
        {"name": "sweep_64", "kind": "batch", "colonies": 64, "low": 500, "high": 20000},
        # The contact graph of a colony for analysis, host arrays both ways.
        {"name": "contacts_100k", "kind": "contacts", "cells": 100003, "margin": 0.1},
        # The wall contacts of a monolayer in a device's chamber.
        {"name": "walls_50k", "kind": "walls", "cells": 50000, "margin": 0.1},
        # A contact system of a caller's own stepper: one solve from zero.
        {"name": "solve_8k", "kind": "solve", "bodies": 8000, "law": "linear"},
        # The index of contacts that are already on the device.
        {"name": "graph_1m", "kind": "graph", "cells": 1000000},
        # One training step of the warm-start network: forward, backward, Adam.
        {"name": "train_8k", "kind": "train", "rows": 8192},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "batch", "contacts", "walls", "solve", "graph", "train"))
    if kind == "step":
        start = rng.choice(("settled", "settled", "random", "flow", "trap"))
        top = {"settled": 700000, "random": 2000, "flow": 200000, "trap": 90000}[start]
        cells = _log(rng, 200, top)
        return {"kind": kind, "cells": cells, "start": start, "resident": cells > 2000 or rng.random() < 0.3,
                "law": rng.choice(("none", "none", "linear", "exponential"))}
    if kind == "batch":
        return {"kind": kind, "colonies": _log(rng, 4, 64), "low": 200, "high": _log(rng, 1000, 20000)}
    if kind in ("contacts", "walls"):
        return {"kind": kind, "cells": _log(rng, 100, 200000), "margin": rng.choice((0.01, 0.1))}
    if kind == "solve":
        return {"kind": kind, "bodies": _log(rng, 200, 40000), "law": rng.choice(tuple(LAWS))}
    if kind == "graph":
        return {"kind": kind, "cells": _log(rng, 1000, 1000000)}
    return {"kind": kind, "rows": _log(rng, 200, 60000)}


# ---- inputs --------------------------------------------------------------


def _tracks(n, seed):
    """Capsules end to end in parallel tracks: centres, directions and
    lengths in track order, and each capsule's track."""
    rng = np.random.default_rng(seed)
    lengths = rng.uniform(2.0, 4.0, n)
    pitch = 2.0 * RADIUS + 0.03
    tracks = max(1, int(round(math.sqrt(n * 4.05 / pitch))))
    track = (np.arange(n, dtype=np.int64) * tracks) // n
    step = lengths + 2.0 * RADIUS + rng.exponential(0.03, n) - 0.01
    end = np.cumsum(step)
    first = np.searchsorted(track, track)  # each track's first capsule
    x = end - 0.5 * step - (end - step)[first] + rng.uniform(-2.0, 2.0, tracks)[track]
    y = track * pitch + rng.normal(0.0, 0.012, n)
    angle = rng.normal(0.0, 0.008, n)
    positions = np.stack([x, y, rng.normal(0.0, 0.003, n)], axis=1)
    directions = np.stack([np.cos(angle), np.sin(angle), rng.normal(0.0, 0.001, n)], axis=1)
    return positions, directions, lengths, track


def settled_colony(n, seed):
    """The tracks' capsules as a WorldState whose slots follow no spatial
    order, as after many divisions."""
    positions, directions, lengths, _ = _tracks(n, seed)
    order = np.random.default_rng(seed + 1).permutation(n)
    rates = np.random.default_rng(seed + 2).uniform(0.8 * GROWTH, 1.2 * GROWTH, n)
    return WorldState.from_arrays(positions[order], directions[order], lengths[order], RADIUS, growth_rates=rates)


def channel_flow(world, seed):
    """A shear flow with a swirl over the colony's box on a planar lattice,
    some sites solid."""
    rng = np.random.default_rng(seed)
    low = (float(world.position_x.min()) - 5.0, float(world.position_y.min()) - 5.0)
    high = (float(world.position_x.max()) + 5.0, float(world.position_y.max()) + 5.0)
    spacing = max(4.0, math.sqrt((high[0] - low[0]) * (high[1] - low[1]) / 40000.0))
    sx, sy = (max(2, int((high[k] - low[k]) / spacing) + 1) for k in (0, 1))
    j = (np.arange(sy) + 0.5) / sy
    speed = 4.0 * spacing * j * (1.0 - j)
    x_faces = np.broadcast_to(speed[None, :, None], (sx + 1, sy, 1)) * rng.uniform(0.9, 1.1, (sx + 1, sy, 1))
    y_faces = 0.1 * spacing * np.sin(np.linspace(0.0, 6.0, sx))[:, None, None] * np.ones((1, sy + 1, 1))
    solid = (rng.random((sx, sy, 1)) < 0.02).astype(np.uint8)
    return FlowField((sx, sy, 1), (low[0], low[1], 0.0), (spacing,) * 3, x_faces.astype(np.float32),
                     y_faces.astype(np.float32), np.zeros((sx, sy, 2), np.float32), solid)


def _neighbours(n, seed):
    """Touching pairs of the tracks' capsules: the next one in the track and
    the nearest one in the next track, with a point and a normal each."""
    positions, directions, lengths, track = _tracks(n, seed)
    a = np.flatnonzero(track[:-1] == track[1:])
    half = 0.5 * lengths[:, None] * directions
    tip = positions[a] + half[a]
    tail = positions[a + 1] - half[a + 1]
    pairs = [(a, a + 1, 0.5 * (tip + tail), tail - tip)]
    width = positions[:, 0].max() - positions[:, 0].min() + 100.0
    key = track * width + (positions[:, 0] - positions[:, 0].min())
    order = np.argsort(key)
    at = np.minimum(np.searchsorted(key[order], key + width), n - 1)
    b = order[at]
    keep = (track[b] == track + 1) & (np.abs(positions[b, 0] - positions[:, 0]) < 0.5 * (lengths[b] + lengths))
    a, b = np.flatnonzero(keep), b[keep]
    middle = 0.5 * (positions[a] + positions[b])
    across = np.zeros_like(middle)
    across[:, 1] = 1.0
    pairs.append((a, b, middle, across))
    first, second, point, normal = (np.concatenate([p[k] for p in pairs]) for k in range(4))
    normal = normal / np.linalg.norm(normal, axis=1, keepdims=True)
    order = np.lexsort((second, first))
    return (first[order], second[order], point[order], normal[order]), (positions, directions, lengths)


def _most(pairs, share, n, seed):
    """A random `share` * n of the pairs, in their order."""
    kept = np.sort(np.random.default_rng(seed + 3).permutation(len(pairs[0]))[:int(share * n)])
    return tuple(p[kept] for p in pairs)


def contact_records(n, seed):
    """Cell contacts in (first id, second id) order of a colony whose slots
    follow no spatial order."""
    first, second, point, normal = _most(_neighbours(n, seed)[0], CONTACTS, n, seed)
    rng = np.random.default_rng(seed + 1)
    slot = rng.permutation(n)
    a, b = slot[first], slot[second]
    swap = a > b
    out = np.zeros(len(a), dtype=abi.CELL_CONTACT_DTYPE)
    out["first_slot"], out["second_slot"] = np.where(swap, b, a), np.where(swap, a, b)
    out["first_id"], out["second_id"] = out["first_slot"] + np.uint64(1), out["second_slot"] + np.uint64(1)
    out["point_on_first"] = point
    out["normal"] = np.where(swap[:, None], -normal, normal)
    out["signed_separation"] = rng.uniform(-0.02, 0.02, len(a))
    out["weight"] = 1.0
    return out[np.lexsort((out["second_id"], out["first_id"]))]


def contact_system(n, seed, law):
    """The rows and bodies of the tracks' capsules growing by 1 %: gaps and
    overlaps of up to 0.02 um, the stepper's mobilities and compliance."""
    pairs, (positions, directions, lengths) = _neighbours(n, seed)
    first, second, point, normal = _most(pairs, CONTACTS, n, seed)
    rng = np.random.default_rng(seed + 1)
    rows, bodies = empty_rows(len(first)), empty_bodies(n)

    def lever(body):
        along = np.einsum("ij,ij->i", directions[body], point - positions[body]) / lengths[body]
        return np.clip(along, -0.5, 0.5) * np.einsum("ij,ij->i", directions[body], normal)

    rows["first_slot"], rows["second_slot"] = first, second
    rows["first_jacobian"] = np.concatenate([-normal, -np.cross(point - positions[first], normal)], axis=1)
    rows["second_jacobian"] = np.concatenate([normal, np.cross(point - positions[second], normal)], axis=1)
    rows["first_length_lever"] = np.maximum(0.0, lever(first))
    rows["second_length_lever"] = np.maximum(0.0, -lever(second))
    rows["offset"] = rng.exponential(0.03, len(first)) - 0.02
    rows["compliance"] = 1.0e-4
    drag = lengths + 2.0 * RADIUS
    bodies["axis"] = directions
    bodies["translational_mobility"] = 1.0 / drag
    bodies["axial_mobility"] = 1.0 / (0.5 * drag * RADIUS * RADIUS)
    bodies["transverse_mobility"] = 12.0 / (drag * (drag * drag + 3.0 * RADIUS * RADIUS))
    bodies["length_rate"] = GROWTH * lengths
    return ContactSystem(rows, bodies, DT, LAWS[law])


# ---- cases ---------------------------------------------------------------


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_step(case, seed):
    n, start = case["cells"], case["start"]
    walls = flow = None
    if start == "random":
        world = workloads.colony_1k(seed, n, side=40.0 * math.sqrt(n / 1000.0), growth_rate=GROWTH)
    elif start == "trap":
        world, walls = workloads.trap_colony(n, seed=seed, growth_rate=GROWTH)
    else:
        world = settled_colony(n, seed)
    dynamics = ContactDynamicsParameters(overlap_tolerance=TOLERANCE, growth=LAWS[case["law"]],
                                         flow_drift=start == "flow")
    simulation = Simulation()
    if start == "flow":
        flow = channel_flow(world, seed)
        simulation.backend.set_flow_field(flow)
    state = {"dynamics": dynamics, "start": world, "walls": walls, "simulation": simulation, "run": _step_host}
    if walls is not None:
        simulation.constraints = walls
    if case["resident"]:
        cells = DeviceCells(world)
        state.update(run=_step_resident, cells=cells, outputs=DeviceOutputs(n),
                     fields=[cells.fields[name] for name in GEOMETRY],
                     saved=[cells.fields[name].clone() for name in GEOMETRY])
    return state


def _step_host(state):
    """One step from the kept start: a program that plays a state forward."""
    simulation = state["simulation"]
    simulation.world = state["start"].copy()
    result = simulation.step(DT, state["dynamics"])
    world = simulation.world
    return {**{name: getattr(world, name) for name in GEOMETRY}, "velocities": result.center_velocities,
            "loads": result.axial_loads, "increments": result.length_increments,
            "substeps": result.report.substeps}


def _step_resident(state):
    """The same with the cells on the device.  The backend works on a stream
    of its own, so a program that edits its tensors waits for its edits."""
    torch._foreach_copy_(state["fields"], state["saved"])
    torch.cuda.synchronize()
    report = state["simulation"].backend.advance_contact_dynamics_device(
        state["cells"], state["walls"], DT, state["dynamics"], outputs=state["outputs"])
    out = state["outputs"]
    return {**dict(zip(GEOMETRY, state["fields"])), "velocities": out.velocities, "loads": out.loads,
            "increments": out.increments, "substeps": report.substeps}


def _prepare_batch(case, seed):
    sizes, stiffness, drag = workloads.sweep_sizes(case["colonies"], case["low"], case["high"])
    defaults = ContactDynamicsParameters()
    batch = ColonyBatch([settled_colony(int(n), seed * 1000 + k) for k, n in enumerate(sizes)],
                        defaults.drag * drag, defaults.contact_stiffness * stiffness)
    cells = DeviceCells(batch.concatenated())
    return {"run": _step_batch, "backend": B200Backend(), "batch": batch, "counts": batch.counts(), "cells": cells,
            "outputs": DeviceOutputs(cells.count), "dynamics": ContactDynamicsParameters(overlap_tolerance=TOLERANCE),
            "fields": [cells.fields[name] for name in GEOMETRY],
            "saved": [cells.fields[name].clone() for name in GEOMETRY]}


def _step_batch(state):
    torch._foreach_copy_(state["fields"], state["saved"])
    torch.cuda.synchronize()
    report, colonies = state["backend"].advance_contact_dynamics_batch(
        state["cells"], state["counts"], state["batch"].drag, state["batch"].stiffness, DT, state["dynamics"],
        outputs=state["outputs"])
    out = state["outputs"]
    return {**dict(zip(GEOMETRY, state["fields"])), "velocities": out.velocities, "loads": out.loads,
            "increments": out.increments, "substeps": report.substeps, "rows": colonies["rows"]}


def _prepare_contacts(case, seed):
    """One of the 16 mirror images of the case's colony: the seed moves every
    capsule, and the contacts' number stays."""
    simulation = Simulation()
    world = settled_colony(case["cells"], case["cells"])
    if seed & 8:
        for a, b in (("position_x", "position_y"), ("direction_x", "direction_y")):
            x, y = getattr(world, a), getattr(world, b)
            setattr(world, a, y)
            setattr(world, b, x)
    for k, axis in enumerate("xyz"):
        if seed & (1 << k):
            for name in ("position_", "direction_"):
                setattr(world, name + axis, -getattr(world, name + axis))
    simulation.world = world
    return {"run": _find_contacts, "simulation": simulation, "parameters": ContactParameters(case["margin"])}


def _find_contacts(state):
    graph = state["simulation"].find_cell_contacts(state["parameters"])
    records = graph.contacts
    return {**{name: records[name] for name in records.dtype.names if name != "reserved"},
            "incidence_offsets": graph.incidence_offsets, "incidence": graph.incidence_contacts,
            "neighbor_offsets": graph.neighbor_offsets, "neighbors": graph.packed_neighbor_ids}


def _prepare_walls(case, seed):
    """A monolayer between a device's floor and ceiling: every capsule within
    the margin of both, the side walls and a post farther off."""
    simulation = Simulation()
    world = settled_colony(case["cells"], seed)
    world.position_z[:] = np.random.default_rng(seed + 4).uniform(-0.001, 0.001, len(world))
    world.direction_x, world.direction_y, world.direction_z = normalized_arrays(
        world.direction_x, world.direction_y, np.zeros_like(world.direction_z))
    simulation.world = world
    walls, gap = simulation.constraints, RADIUS + 0.005
    walls.add_plane(point=(0.0, 0.0, -gap), inward_normal=(0.0, 0.0, 1.0))
    walls.add_plane(point=(0.0, 0.0, gap), inward_normal=(0.0, 0.0, -1.0))
    low = [float(getattr(world, name).min()) - 5.0 for name in ("position_x", "position_y")]
    high = [float(getattr(world, name).max()) + 5.0 for name in ("position_x", "position_y")]
    middle, half = [0.5 * (a + b) for a, b in zip(low, high)], [0.5 * (b - a) for a, b in zip(low, high)]
    walls.add_box(center=(*middle, 0.0), half_extents=(*half, 3.0), allowed_region=abi.REGION_INSIDE)
    walls.add_cylinder(center=(low[0] - 10.0, middle[1], 0.0), radius=5.0, half_height=3.0)
    return {"run": _find_walls, "simulation": simulation, "parameters": ConstraintContactParameters(case["margin"])}


def _find_walls(state):
    graph = state["simulation"].find_external_contacts(state["parameters"])
    records = graph.contacts
    return {**{name: records[name] for name in records.dtype.names if name != "reserved"},
            "incidence_offsets": graph.incidence_offsets, "incidence": graph.incidence_contacts}


def _prepare_solve(case, seed):
    system = contact_system(case["bodies"], seed, case["law"])
    return {"run": _solve, "backend": B200Backend(), "system": system,
            "zero": np.zeros(len(system.rows), dtype=np.float32),
            "parameters": ContactSolveParameters(0.25 * TOLERANCE)}


def _solve(state):
    backend, system = state["backend"], state["system"]
    solved = backend.solve_contact_forces(system, state["zero"], state["parameters"])
    response = backend.evaluate_contact_response(system, solved.multipliers)
    return {"multipliers": solved.multipliers, "velocities": response.velocities, "loads": response.loads,
            "rates": response.length_rates, "status": solved.report.status}


def _prepare_graph(case, seed):
    records = contact_records(case["cells"], seed)
    contacts = torch.from_numpy(records.view(np.uint8).copy()).cuda()
    index, tensors = device_index(case["cells"], 2 * len(records), "cuda:0")
    return {"run": _build_graph, "backend": B200Backend(), "contacts": contacts, "count": len(records),
            "cells": case["cells"], "index": index, "tensors": tensors}


def _build_graph(state):
    total = state["backend"].build_contact_graph_device(state["contacts"].data_ptr(), state["count"], state["cells"],
                                                        state["index"])
    tensors = state["tensors"]
    return {**{name: tensors[name] for name in tensors if name != "neighbor_ids"},
            "neighbor_ids": tensors["neighbor_ids"][:total]}


def _training_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((case["rows"], learned.INPUT), dtype=np.float32)
    x[:, :learned.FEATURES] = rng.uniform(-1.0, 1.0, (case["rows"], learned.FEATURES))
    return learned.to_bf16_bits(x), rng.normal(0.0, 1.0, (case["rows"], learned.OUTPUTS)).astype(np.float32)


def _prepare_train(case, seed):
    x, y = _training_inputs(case, seed)
    net = learned.WarmStartNetwork("cuda:0", seed=seed)
    return {"run": _train, "net": net, "features": torch.from_numpy(x.view(np.int16)).cuda(),
            "targets": torch.from_numpy(y).cuda(),
            "kept": [(t, t.clone()) for t in (net.params, net.m, net.v, net.weights, net.biases)]}


def _train(state):
    """One step of WarmStartNetwork.train from the kept parameters."""
    net = state["net"]
    for tensor, start in state["kept"]:
        tensor.copy_(start)
    net.step = 0
    outputs, activations = net.forward(state["features"], keep=True)
    diff, factor = net.loss_and_grad(outputs, state["targets"])
    grads = net.backward(state["features"], activations, (diff * factor).contiguous())
    net.adam(2e-3)
    return {"outputs": outputs, "grads": grads, "params": net.params}


# ---- what a pass cannot do without, and how close results have to be ------


def _rows_of(case):
    return int(CONTACTS * case.get("cells", case.get("bodies", 0)))


def work(case):
    kind = case["kind"]
    if kind == "step":  # ids, geometry, growth and flags in; geometry and outputs out
        return {"bytes": case["cells"] * (45 + 48), "flops": 0}
    if kind == "batch":
        low, high = math.log(case["low"]), math.log(case["high"])
        mean = (case["high"] - case["low"]) / (high - low)
        return {"bytes": case["colonies"] * mean * (45 + 48), "flops": 0}
    if kind == "contacts":  # records, and an index of two entries a contact
        return {"bytes": case["cells"] * (45 + 16) + _rows_of(case) * (64 + 32), "flops": 0}
    if kind == "walls":  # two contacts a capsule with the floor and two with the ceiling
        return {"bytes": case["cells"] * (45 + 8 + 4 * (64 + 8)), "flops": 0}
    if kind == "solve":  # the system in twice, multipliers and response out
        return {"bytes": 2 * (case["bodies"] * 52 + _rows_of(case) * 72) + case["bodies"] * 32 + _rows_of(case) * 4,
                "flops": 0}
    if kind == "graph":
        return {"bytes": _rows_of(case) * (64 + 32) + case["cells"] * 16, "flops": 0}
    macs = sum(o * k for o, k in learned.W_SHAPES)
    return {"bytes": case["rows"] * (2 * learned.INPUT + 4 * 2 * learned.OUTPUTS) + 4 * 7 * learned.PARAMETERS,
            "flops": 6.0 * case["rows"] * macs}


def tolerance(case):
    kind = case["kind"]
    if kind in ("step", "batch"):
        # FP32 iterates of the relaxation, whose step lengths are FP64 sums
        # rounded to FP32.  The two forms of set_relaxation sum in different
        # orders and gave the same bits in every listed case; a step length
        # that does round the other way moves the iterate within the solve's
        # tolerance (1.25e-4 um of the 0.1 um that cells move in a step).
        return {"rel": 1e-4, "max": 0.05, "differ": 0.0}
    if kind in ("contacts", "walls"):
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}  # FP32 geometry, no sums to reorder
    if kind == "solve":
        return {"rel": 1e-4, "max": 0.05, "differ": 0.0}
    if kind == "graph":
        return "exact"
    return {"rel": 1e-2, "max": 0.1}  # bf16 activations


def exact(case, seed):
    kind = case["kind"]
    if kind == "step" and case["law"] == "none" and case["cells"] <= 200000:
        # Without a load law a cell's length grows by rate * length * dt
        # whatever touches it; the rest of a step is an iterate within the
        # overlap tolerance, which no 64-bit value pins.
        state_free = _start_world(case, seed)
        length = state_free.lengths.astype(np.float64)
        increment = state_free.growth_rates.astype(np.float64) * length * DT
        return {**{name: None for name in GEOMETRY}, "lengths": length + increment, "velocities": None,
                "loads": None, "increments": increment, "substeps": None}
    if kind == "train":
        return _train_exact(case, seed)
    return None


def _start_world(case, seed):
    n = case["cells"]
    if case["start"] == "random":
        return workloads.colony_1k(seed, n, side=40.0 * math.sqrt(n / 1000.0), growth_rate=GROWTH)
    if case["start"] == "trap":
        return workloads.trap_colony(n, seed=seed, growth_rate=GROWTH)[0]
    return settled_colony(n, seed)


def _train_exact(case, seed):
    """The same step in 64 bits on the bf16 weights and features given."""
    bits, y = _training_inputs(case, seed)
    x = torch.from_numpy((bits.astype(np.uint32) << 16).view(np.float32)).double()
    p = learned.initial_parameters(seed)
    w = (learned.to_bf16_bits(p[:learned.WEIGHTS]).astype(np.uint32) << 16).view(np.float32)
    layers, at = [], 0
    for i, (o, k) in enumerate(learned.W_SHAPES):
        bias_at = learned.WEIGHTS + i * learned.HIDDEN
        layers.append((torch.from_numpy(w[at:at + o * k].reshape(o, k)).double().requires_grad_(),
                       torch.from_numpy(p[bias_at:bias_at + o]).double().requires_grad_()))
        at += o * k
    h = x
    for i, (weight, bias) in enumerate(layers):
        h = h @ weight.T + bias
        if i < 3:
            h = torch.nn.functional.gelu(h)
    outputs = h[:, :learned.OUTPUTS]
    diff = outputs - torch.from_numpy(y).double()
    (diff * diff).mean().backward()
    grads = torch.cat([weight.grad.reshape(-1) for weight, _ in layers] + [bias.grad for _, bias in layers])
    # Adam's first step from zero moments divides the gradient by its own
    # size, so a weight whose gradient is rounding noise has no 64-bit value.
    return {"outputs": outputs.detach(), "grads": grads, "params": None}
