"""The work that users of this framework have it do, as timed cases.

A case is one pass of a program that is already set up: a network advanced by some
milliseconds of biological time through `mb.run`, or the spike-output surrogate network
trained or evaluated.  The networks are those of mind_b200.networks (ball-and-stick cells
with ExpSyn; random binary trees and pyramidal cells in recurrent Exp2Syn networks;
pyramidal cells coupled to Jansen-Rit regions), built here through the public builders from
a seed, with cells in populations that share a morphology.  A pass continues the
simulation from where the last one stopped and returns what a user records: the somas' and
one dendritic voltage per cell, the raster, and the regions' outputs.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mind.jl_b200"))

import mind_b200 as mb  # noqa: E402
from mind_b200 import surrogate  # noqa: E402
from mind_b200.macro import MacroModel  # noqa: E402

DT = 0.025              # ms
MORPHOLOGIES = 48       # distinct morphologies in a network of trees or pyramids
FEATURES = surrogate.N_FEATURES


def listed():
    return [
        # one neuron stepped for a millisecond: a closed loop or an interactive session,
        # where launches and the latency of one cell are everything
        {"name": "stick_1_fp64", "kind": "network", "family": "stick", "cells": 1, "synapses": 10,
         "precision": "fp64", "steps": 40},
        # the ball-and-stick benchmark network, 10 ms
        {"name": "stick_64_fp64", "kind": "network", "family": "stick", "cells": 64, "synapses": 10,
         "precision": "fp64", "steps": 400},
        # a small network of uneven trees: fewer cells than the GPU has multiprocessors
        {"name": "trees_61_fp64", "kind": "network", "family": "trees", "cells": 61, "synapses": 100,
         "precision": "fp64", "steps": 397},
        # a large network of uneven trees, many more cells than fit on the chip at once
        {"name": "trees_4000_fp64", "kind": "network", "family": "trees", "cells": 4000, "synapses": 100,
         "precision": "fp64", "steps": 200},
        # the same in the mixed mode (FP32 gating, FP64 cable), an ordinary size
        {"name": "trees_1500_mixed", "kind": "network", "family": "trees", "cells": 1500, "synapses": 100,
         "precision": "mixed", "steps": 400},
        # pyramidal cells (700-1,200 compartments, 300 synapses) in a dense recurrent network
        {"name": "pyramids_250_fp64", "kind": "network", "family": "pyramids", "cells": 250, "synapses": 300,
         "precision": "fp64", "steps": 200},
        # the pyramidal network at its benchmark size
        {"name": "pyramids_1000_mixed", "kind": "network", "family": "pyramids", "cells": 1000, "synapses": 300,
         "precision": "mixed", "steps": 200},
        # a voltage-clamp experiment: SEClamp electrodes, which run as code emitted from MOD files
        {"name": "clamped_151_fp64", "kind": "network", "family": "clamped", "cells": 151, "synapses": 300,
         "precision": "fp64", "steps": 200},
        # pyramidal cells coupled to neural-mass regions
        {"name": "regions_600_mixed", "kind": "regions", "cells": 600, "populations": 20, "synapses": 300,
         "precision": "mixed", "steps": 400},
        # the same coupling with the surrogate network standing in for 98% of the cells
        {"name": "surrogate_1000_mixed", "kind": "surrogate", "cells": 1000, "populations": 20, "synapses": 300,
         "precision": "mixed", "steps": 400},
        # training the surrogate: Adam steps of 4,096 windows
        {"name": "train_4096", "kind": "train", "rows": 8192, "batch": 4096, "steps": 40},
        # evaluating the surrogate on recorded windows
        {"name": "predict_20000", "kind": "predict", "rows": 20000},
    ]


def _spread(rng, low, high):
    """A whole number spread over [low, high] by its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["stick", "trees", "trees", "pyramids", "pyramids", "clamped", "regions", "surrogate", "train",
                       "predict"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "stick":
        return {"kind": "network", "family": kind, "cells": _spread(rng, 1, 300), "synapses": rng.randint(1, 20),
                "precision": precision, "steps": _spread(rng, 40, 500)}
    if kind == "trees":
        return {"kind": "network", "family": kind, "cells": _spread(rng, 3, 2000), "synapses": rng.randint(20, 120),
                "precision": precision, "steps": _spread(rng, 100, 400)}
    if kind in ("pyramids", "clamped"):
        return {"kind": "network", "family": kind, "cells": _spread(rng, 3, 700), "synapses": rng.randint(50, 320),
                "precision": precision, "steps": _spread(rng, 60, 300)}
    if kind in ("regions", "surrogate"):
        populations = rng.randint(2, 24)
        return {"kind": kind, "cells": populations * _spread(rng, 4, 40), "populations": populations,
                "synapses": rng.randint(32, 300), "precision": precision, "steps": 40 * rng.randint(3, 10)}
    if kind == "train":
        return {"kind": kind, "rows": _spread(rng, 500, 8000), "batch": _spread(rng, 100, 4096),
                "steps": rng.randint(5, 40)}
    return {"kind": kind, "rows": _spread(rng, 50, 19000)}


# ---------------------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------------------

def _soma():
    return mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0)


def _tree(rng, compartments):
    """A random binary dendritic tree of `compartments` compartments of 10 um (branches
    lognormal around 50 um, diameters tapering 0.9x from 3 um)."""
    sections, leaves, budget = [_soma()], [("soma", 3.0 / 0.9)], compartments
    while budget > 0:
        parent, diameter = leaves.pop(int(rng.integers(len(leaves))))
        for _ in range(1 if parent == "soma" else 2):
            if budget <= 0:
                break
            nseg = min(budget, max(1, int(round(rng.lognormal(math.log(50.0), 0.5) / 10.0))))
            budget -= nseg
            name = "d%d" % len(sections)
            sections.append(mb.Section(name, label="dend", parent=parent, parent_x=1.0, length=10.0 * nseg,
                                       diameter=diameter * 0.9, nseg=nseg, Ra=100.0, cm=1.0))
            leaves.append((name, diameter * 0.9))
    return sections


def _pyramid(rng, compartments):
    """A pyramidal cell: a 600 um apical trunk with 10-20 obliques and 5-10 tuft branches, and
    4-8 basal dendrites of 150-250 um; hh goes on the soma and the proximal 100 um."""
    d = rng.uniform(2.5, 4.0)
    sections = [_soma(),
                mb.Section("trunk0", label="prox", parent="soma", parent_x=1.0, length=100.0, diameter=d, nseg=10),
                mb.Section("trunk1", label="apical", parent="trunk0", parent_x=1.0, length=500.0, diameter=0.6 * d,
                           nseg=50)]
    left = compartments - 61
    for b in range(int(rng.integers(4, 9))):
        nseg = int(rng.integers(15, 26))
        d = rng.uniform(0.8, 2.0)
        sections.append(mb.Section("basal%dp" % b, label="prox", parent="soma", parent_x=0.0, length=100.0, diameter=d,
                                   nseg=10))
        sections.append(mb.Section("basal%dd" % b, label="basal", parent="basal%dp" % b, parent_x=1.0,
                                   length=10.0 * (nseg - 10), diameter=0.8 * d, nseg=nseg - 10))
        left -= nseg
    oblique, tuft = int(rng.integers(10, 21)), int(rng.integers(5, 11))
    shares = rng.dirichlet(np.ones(oblique + tuft)) * max(left, oblique + tuft)
    for k, share in enumerate(shares):
        nseg = max(1, int(round(share)))
        x = rng.uniform(0.05, 0.95) if k < oblique else 1.0
        sections.append(mb.Section("ap%d" % k, label="apical", parent="trunk1", parent_x=float(x), length=10.0 * nseg,
                                   diameter=rng.uniform(0.6, 1.5), nseg=nseg))
    return sections


def _cells(model, rng, family, count):
    """`count` cells in populations that share a morphology; per cell (cell, dendritic sections)."""
    kinds = 1 if family == "stick" else min(count, MORPHOLOGIES)
    sizes = {"trees": (100, 1000), "pyramids": (700, 1200), "clamped": (700, 1200), "small": (300, 600)}.get(family)
    out = []
    for k in range(kinds):
        if family == "stick":
            secs = [_soma(), mb.Section("dend", label="dend", parent="soma", parent_x=1.0, length=500.0, diameter=2.0,
                                        nseg=50, Ra=100.0, cm=1.0)]
        else:
            size = int(round(sizes[0] + (sizes[1] - sizes[0]) * (k + rng.uniform()) / kinds))
            secs = _tree(rng, size - 1) if family == "trees" else _pyramid(rng, size)
        n = count // kinds + (k < count % kinds)
        rest = rng.uniform(-70.0, -60.0, n)
        for cell in mb.add_population(model, secs, n, voltage=lambda i: float(rest[i - 1])):
            active = [s.label for s in secs if s.label in ("soma", "prox")]
            mb.insert(cell, mb.builtin("hh"), sections=sorted(set(active)))
            mb.insert(cell, mb.builtin("pas"), sections=sorted({s.label for s in secs} - set(active)),
                      params={"g": 1.0e-4, "e": -65.0})
            mb.register_spike_source(cell, threshold=-10.0)
            out.append((cell, secs[1:]))
    return out


def _synapses(model, rng, family, cells, per_cell):
    """`per_cell` synapses at random dendritic places of every cell; returns the first point."""
    owners = np.repeat([c.index for c, _ in cells], per_cell)
    xs = rng.uniform(0.0, 1.0, len(owners))
    if family == "stick":
        return mb.add_pointprocesses(model, mb.builtin("ExpSyn"), owners, "dend", xs, {"tau": 2.0, "e": 0.0})
    names = []
    for _, dends in cells:
        w = np.array([s.nseg for s in dends], dtype=float)
        names += [dends[i].name for i in rng.choice(len(dends), size=per_cell, p=w / w.sum())]
    e = np.where(rng.uniform(size=len(owners)) < 0.8, 0.0, -80.0)
    return mb.add_pointprocesses(model, mb.builtin("Exp2Syn"), owners, names, xs, {"tau1": 0.5, "tau2": 5.0, "e": e})


def _weights(rng, n):
    return rng.lognormal(math.log(0.4), 0.6, n) / 1000.0   # uS


def _recurrent(model, rng, family, cells, first, per_cell):
    """NetCons between the cells: one per synapse on trees, 3% connectivity on pyramids."""
    n = len(cells)
    if family == "stick" or n < 2:
        return
    each = per_cell if family == "trees" else max(1, int(round(0.03 * n)))
    low, high = (1.0, 5.0) if family == "trees" else (0.5, 3.0)
    targets = first + np.repeat(np.arange(n) * per_cell, each) + rng.integers(0, per_cell, n * each)
    mb.connect_many(model, rng.integers(1, n + 1, n * each), targets, _weights(rng, n * each),
                    rng.uniform(low, high, n * each))


def _network(case, seed):
    """The built model of a network case."""
    rng = np.random.default_rng([seed, 1])
    family, n, per_cell = case["family"], case["cells"], case["synapses"]
    model = mb.MicroModel(celsius=6.3)
    cells = _cells(model, rng, family, n)
    first = _synapses(model, rng, family, cells, per_cell)
    _recurrent(model, rng, family, cells, first, per_cell)
    # every synapse has its own Poisson background: 10 Hz on the sticks, 5 Hz on trees, 2 Hz on pyramids
    total = n * per_cell
    rate = {"stick": 10.0, "trees": 5.0}.get(family, 2.0)
    stims = mb.add_pointprocesses(model, mb.builtin("NetStim"), np.zeros(total, np.int64), "none", np.zeros(total),
                                  {"interval": 1000.0 / rate, "number": 1e9, "start": 0.0, "noise": 1.0})
    sources = mb.register_point_sources(model, np.arange(stims, stims + total))
    mb.connect_many(model, sources, np.arange(first, first + total), _weights(rng, total), np.zeros(total))
    if family in ("pyramids", "clamped"):
        chosen = np.arange(1, max(1, n // 10) + 1)
        mb.add_pointprocesses(model, mb.builtin("IClamp"), chosen, "soma", np.full(len(chosen), 0.5),
                              {"del": 1.0, "dur": 50.0, "amp": 0.1})
    if family == "clamped":
        held = np.arange(max(1, n // 10) + 1, n + 1, 3) if n > 2 else np.array([n])
        mb.add_pointprocesses(model, mb.builtin("SEClamp"), held, "soma", np.full(len(held), 0.5),
                              {"rs": 1.0, "dur1": 2.0, "amp1": -65.0, "dur2": 1.0e9, "amp2": -50.0})
    mb.build(model, dt_micro=DT, seed=1 + seed % (1 << 30))
    return model, cells


def _coupled(case, seed):
    """The built model of a network coupled to regions, every synapse driven by its
    population's region, every population's spike rate feeding its region."""
    rng = np.random.default_rng([seed, 2])
    n, per_cell, populations = case["cells"], case["synapses"], case["populations"]
    model = mb.MicroModel(celsius=6.3)
    cells = _cells(model, rng, "small", n)
    order = rng.permutation(n)
    first = _synapses(model, rng, "small", cells, per_cell)
    _recurrent(model, rng, "small", cells, first, per_cell)
    inputs = mb.register_external_sources(model, n * per_cell)
    mb.connect_many(model, inputs, np.arange(first, first + n * per_cell), _weights(rng, n * per_cell),
                    np.zeros(n * per_cell))
    macro = MacroModel(dt_macro=0.1, bin_ms=1.0)
    for _ in range(populations):
        macro.add_region(micro_gain=1.0)
    for src in range(1, populations + 1):
        for dst in range(1, populations + 1):
            if src != dst and rng.uniform() < 0.2:
                macro.connect(src, dst, float(rng.uniform(0.0, 1.0)), int(rng.integers(1, 21)))
    for rank, c in enumerate(order):
        region = rank * populations // n + 1
        macro.add_inputs(region, inputs[c * per_cell:(c + 1) * per_cell], 2.0)
        macro.add_outputs(region, [c + 1])     # detector of cell c is source c + 1
    model.macro = macro
    mb.build(model, dt_micro=DT, seed=1 + seed % (1 << 30))
    return model, cells


def _records(model, cells):
    """The soma and the end of one dendrite of every cell."""
    out = [mb.voltage_record(model, c) for c, _ in cells]
    return out + [mb.voltage_record(model, c, section=dends[-1].name, x=0.9, name="dend_%d" % c.gid)
                  for c, dends in cells]


def _raster_size(case):
    """Room for a pass's spikes: twice the background's, and every cell firing every 4 ms."""
    n, ms = case["cells"], case["steps"] * DT
    rate = {"stick": 10.0, "trees": 5.0, "pyramids": 2.0, "clamped": 2.0}.get(case.get("family"), 0.0)
    return 64 + int(2.0 * n * case["synapses"] * rate * ms / 1000.0 + n * ms / 4.0)


# ---------------------------------------------------------------------------------------
# the surrogate network's data: 20 ms of binned synaptic drive and 5 ms of own spikes
# ---------------------------------------------------------------------------------------

def _windows(rows, seed):
    rng = np.random.default_rng([seed, 3])
    x = np.zeros((rows, FEATURES), dtype=np.float32)
    busy = rng.uniform(size=x.shape) < 0.15
    x[busy] = rng.exponential(1.0, int(busy.sum())).astype(np.float32)
    x[:, 640:] = rng.uniform(size=(rows, FEATURES - 640)) < 0.03
    y = (rng.uniform(size=rows) < 0.03 + 0.2 * (x[:, :640].mean(axis=1) > 0.16)).astype(np.float32)
    return x, y


def prepare(case, seed):
    if case["kind"] in ("train", "predict"):
        x, y = _windows(case["rows"], seed)
        return {"case": case, "net": surrogate.Mlp(seed=1 + seed % 1000), "x": x, "y": y}
    model, cells = (_network if case["kind"] == "network" else _coupled)(case, seed)
    mb.initialize(model, case["precision"])
    state = {"case": case, "model": model, "records": _records(model, cells), "spikes": _raster_size(case)}
    if case["kind"] == "surrogate":
        net = surrogate.Mlp(seed=1 + seed % 1000)
        params = net.params
        params[-1] = math.log(0.005 / 0.995)     # about 5 Hz
        net.params = params
        mask = np.random.default_rng([seed, 4]).uniform(size=case["cells"]) >= 0.02
        model.state.attach_surrogate(net, mask, 500.0)
        mb.initialize(model, case["precision"])
        state["net"] = net
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        losses, _ = state["net"].train(state["x"], state["y"], steps=case["steps"], batch=case["batch"], lr=1e-3)
        return {"losses": losses, "params": state["net"].params}
    if case["kind"] == "predict":
        return {"probability": state["net"].predict(state["x"])}
    model = state["model"]
    result = mb.run(model, mb.simulation_time(model) + case["steps"] * DT, records=state["records"])
    times, sids = np.full(state["spikes"], -1.0), np.zeros(state["spikes"], dtype=np.int64)
    n = min(len(times), len(result.spike_times))
    times[:n], sids[:n] = result.spike_times[:n], result.spike_sources[:n]
    out = {"voltage": result.traces.by_record, "times": times, "sids": sids}
    if result.macro_trace is not None:
        out["regions"] = result.macro_trace
    return out


def work(case):
    """One pass: the model and its inputs read once, the recorded outputs and the state
    written once, and the arithmetic of every step or row."""
    if case["kind"] in ("train", "predict"):
        rows = case["rows"]
        flops = 2.0 * (FEATURES * 256 + 2 * 256 * 256 + 256)
        params = 4.0 * (flops / 2 + 3 * 256 + 1)
        if case["kind"] == "predict":
            return {"bytes": rows * (4.0 * FEATURES + 4) + params, "flops": rows * flops}
        return {"bytes": rows * (4.0 * FEATURES + 4) + 2 * params + 4.0 * case["steps"],
                "flops": 3.0 * flops * case["batch"] * case["steps"]}
    n, steps = case["cells"], case["steps"]
    detailed = n if case["kind"] == "network" else n * (0.02 if case["kind"] == "surrogate" else 1.0)
    nodes = {"stick": 54, "trees": 640, "pyramids": 1000, "clamped": 1000}.get(case.get("family"), 480) * detailed
    active = {"stick": 1, "trees": 1}.get(case.get("family"), 71) * detailed
    synapses = case["synapses"] * detailed
    # per node: voltage read and written, axial, capacitance and diagonal terms, leak; per row: its state and parameters
    size = nodes * 64.0 + active * 104.0 + synapses * 68.0 + 2.0 * n * (steps + 1) * 8.0
    # per node: leak, assembly, elimination, back-substitution; per hh row: three gates' rates
    flops = steps * (nodes * 30.0 + active * 180.0 + synapses * 14.0)
    if case["kind"] == "surrogate":
        flops += steps / 40.0 * n * 2.0 * (FEATURES * 256 + 2 * 256 * 256 + 256)
    return {"bytes": size, "flops": flops}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, in plain numpy and torch
# ---------------------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] in ("train", "predict"):
        return _exact_surrogate(case, seed)
    if case["kind"] != "network" or case["family"] == "clamped":
        return None
    if case["steps"] * work(dict(case, steps=0))["bytes"] > 8.0e9:     # would take minutes
        return None
    model, cells = _network(case, seed)
    layout = model.layout
    nodes = [r.node - 1 for r in _records(model, cells)]
    return {"voltage": _exact_run(layout, case["steps"], nodes), "times": None, "sids": None}


def _philox(counter, key):
    """Philox4x32-10 of four 32-bit counter words (arrays) under two key words."""
    c = [np.asarray(x, dtype=np.uint64) for x in counter]
    k0, k1 = key
    low = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p, q = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(q >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), q & low, (p >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _stim_times(layout, end):
    """Firing times up to `end` of every NetStim (exponential intervals from time 0): (time, point)."""
    group = layout.group("NetStim")
    interval = group.column("interval")
    ids = group.logical_ids
    points = np.empty(group.rows, dtype=np.int64)
    g = next(i for i, x in enumerate(layout.groups) if x is group) + 1
    mine = np.flatnonzero(layout.point_group == g)
    points[layout.point_row[mine] - 1] = mine + 1
    key = (layout.seed & 0xFFFFFFFF, layout.seed >> 32)
    third = np.full(len(ids), group.mechanism.digest & 0xFFFFFFFF, dtype=np.uint64)
    low = np.uint64(0xFFFFFFFF)
    t, times, owners, k = np.zeros(len(ids)), [], [], 0
    while True:
        word = _philox((np.full(len(ids), k >> 2, dtype=np.uint64), third, ids & low, ids >> np.uint64(32)), key)[k & 3]
        t = t - interval * np.log((word.astype(np.float64) + 1.0) / (2.0 ** 32 + 1.0))
        live = t <= end
        if not live.any():
            return np.concatenate(times) if times else t[live], np.concatenate(owners) if owners else points[live]
        times.append(t[live])
        owners.append(points[live])
        k += 1


def _exact_run(layout, steps, record):
    dt = layout.dt
    v = layout.voltage.copy()
    parent = layout.parent.astype(np.int64) - 1
    depth = np.zeros(len(v), dtype=np.int64)      # every parent comes before its children
    for i in np.flatnonzero(parent >= 0):
        depth[i] = depth[parent[i]] + 1
    levels = [np.flatnonzero(depth == d) for d in range(depth.max() + 1)]
    child = np.flatnonzero(parent >= 0)
    a, base = layout.axial, layout.capacitance / dt + layout.axial_diagonal

    def rates(u):
        def trap(x, y):
            return np.where(np.abs(x / y) < 1e-6, y * (1.0 - x / y / 2.0), x / np.expm1(np.where(x == 0.0, 1.0, x) / y))
        m = 0.1 * trap(-(u + 40.0), 10.0), 4.0 * np.exp(-(u + 65.0) / 18.0)
        h = 0.07 * np.exp(-(u + 65.0) / 20.0), 1.0 / (np.exp(-(u + 35.0) / 10.0) + 1.0)
        n = 0.01 * trap(-(u + 55.0), 10.0), 0.125 * np.exp(-(u + 65.0) / 80.0)
        return [(p / (p + q), p + q) for p, q in (m, h, n)]

    names = [g.mechanism.name for g in layout.groups]
    node = {g.mechanism.name: g.nodes.astype(np.int64) - 1 for g in layout.groups}
    col = {g.mechanism.name: g.column for g in layout.groups}
    hh = node["hh"]
    q10 = 3.0 ** ((layout.celsius - 6.3) / 10.0)
    gates = [inf for inf, _ in rates(v[hh])]
    kind = "Exp2Syn" if "Exp2Syn" in names else "ExpSyn"
    syn = node[kind]
    if kind == "Exp2Syn":
        t1, t2 = col[kind]("tau1"), col[kind]("tau2")
        peak = t1 * t2 / (t2 - t1) * np.log(t2 / t1)
        factor = 1.0 / (np.exp(-peak / t2) - np.exp(-peak / t1))
        rise = np.zeros(len(syn))
    else:
        t2, factor = col[kind]("tau"), 1.0
    fall = np.zeros(len(syn))
    events = {}       # delivery step -> (synapse rows, weights) lists

    def fire(sources, times):
        """NetCon events of `sources` (0-based) firing at `times`."""
        for s, t in zip(sources, times):
            e = np.arange(layout.fanout_offsets[s] - 1, layout.fanout_offsets[s + 1] - 1)
            rows = layout.point_row[layout.edge_targets[e] - 1] - 1
            steps_at = np.maximum(0, np.ceil((t + layout.edge_delays[e] - 0.5 * dt) / dt)).astype(np.int64)
            for k, r, w in zip(steps_at, rows, layout.edge_weights[e]):
                events.setdefault(int(k), []).append((r, w))

    source_of = np.full(len(layout.point_group) + 1, -1)
    fed = layout.source_points > 0
    source_of[layout.source_points[fed]] = np.flatnonzero(fed)
    times, points = _stim_times(layout, steps * dt)
    fire(source_of[points], times)
    detectors = np.flatnonzero(layout.source_nodes > 0)
    watch, above = layout.source_nodes[detectors] - 1, np.zeros(len(detectors), dtype=bool)
    out = np.empty((len(record), steps + 1))
    out[:, 0] = v[record]
    x = np.zeros(len(v))
    for k in range(steps):
        now = v[watch] > layout.source_thresholds[detectors]
        fire(detectors[now & ~above], np.full(int((now & ~above).sum()), k * dt + 1.0e-10))
        above = now
        for r, w in events.pop(k, ()):
            fall[r] += w * (factor if np.isscalar(factor) else factor[r])
            if kind == "Exp2Syn":
                rise[r] += w * factor[r]
        d, rhs = base.copy(), np.zeros(len(v))
        for name in names:
            i = node[name]
            if name == "pas":
                s, g = layout.area[i] * 0.01, col[name]("g")
                np.add.at(d, i, s * g)
                np.subtract.at(rhs, i, s * g * (v[i] - col[name]("e")))
            elif name == "hh":
                s, (m, h, n) = layout.area[i] * 0.01, gates
                gna, gk, gl = col[name]("gnabar") * m ** 3 * h, col[name]("gkbar") * n ** 4, col[name]("gl")
                np.add.at(d, i, s * (gna + gk + gl))
                np.subtract.at(rhs, i, s * (gna * (v[i] - col[name]("ena")) + gk * (v[i] - col[name]("ek"))
                                            + gl * (v[i] - col[name]("el"))))
            elif name == kind:
                g = fall - rise if kind == "Exp2Syn" else fall
                np.add.at(d, i, g)
                np.subtract.at(rhs, i, g * (v[i] - col[name]("e")))
            elif name == "IClamp":
                t = (k + 0.5) * dt
                on = (t >= col[name]("del")) & (t < col[name]("del") + col[name]("dur"))
                np.add.at(rhs, i, np.where(on, col[name]("amp"), 0.0))
        flow = a[child] * (v[parent[child]] - v[child])
        rhs[child] += flow
        np.subtract.at(rhs, parent[child], flow)
        for i in levels[:0:-1]:
            f = a[i] / d[i]
            np.subtract.at(d, parent[i], f * a[i])
            np.add.at(rhs, parent[i], f * rhs[i])
        x[levels[0]] = rhs[levels[0]] / d[levels[0]]
        for i in levels[1:]:
            x[i] = (rhs[i] + a[i] * x[parent[i]]) / d[i]
        v += x
        gates = [s - np.expm1(-dt * q10 * total) * (inf - s) for s, (inf, total) in zip(gates, rates(v[hh]))]
        fall *= np.exp(-dt / t2)
        if kind == "Exp2Syn":
            rise *= np.exp(-dt / t1)
        out[:, k + 1] = v[record]
    return out


def _exact_surrogate(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    x, y = _windows(case["rows"], seed)
    net = surrogate.Mlp(seed=1 + seed % 1000)      # the initial parameters are an input
    flat = torch.tensor(net.params, dtype=torch.float64, device=device)
    net.close()
    dims = [FEATURES, 256, 256, 256, 1]
    x = torch.tensor(x, dtype=torch.float64, device=device)
    y = torch.tensor(y, dtype=torch.float64, device=device)

    def logits(p, rows):
        at, h = 0, rows
        for i, o in zip(dims[:-1], dims[1:]):
            w, b = p[at:at + i * o].view(o, i), p[at + i * o:at + i * o + o]
            at += i * o + o
            h = h @ w.T + b
            h = torch.nn.functional.silu(h) if o > 1 else h
        return h[:, 0]

    if case["kind"] == "predict":
        return {"probability": torch.sigmoid(logits(flat, x)).cpu().numpy()}
    m1, m2, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    slots = np.arange(case["batch"], dtype=np.uint64)
    for t in range(1, case["steps"] + 1):
        with np.errstate(over="ignore"):            # the batch of step t: a 64-bit mix of step and slot
            s = (np.uint64(t) * np.uint64(0x9E3779B97F4A7C15) + slots * np.uint64(0xBF58476D1CE4E5B9)
                 + np.uint64(0x94D049BB133111EB))
            s ^= s >> np.uint64(31)
            s *= np.uint64(0xD6E8FEB86659FD93)
            s ^= s >> np.uint64(32)
        rows = torch.tensor((s % np.uint64(case["rows"])).astype(np.int64), device=device)
        p = flat.clone().requires_grad_(True)
        loss = torch.nn.functional.binary_cross_entropy_with_logits(logits(p, x[rows]), y[rows])
        (g,) = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        m1 = 0.9 * m1 + 0.1 * g
        m2 = 0.999 * m2 + 0.001 * g * g
        flat = flat - 1e-3 * (m1 / (1 - 0.9 ** t)) / (torch.sqrt(m2 / (1 - 0.999 ** t)) + 1e-8)
    return {"losses": np.array(losses), "params": flat.cpu().numpy()}
