"""The cable solve at the edges of its quotients' range and of its schedules, against the oracle.

The FP64 mode forms its quotients by FMA where every operand lies in a middle range, and
divides a step's whole system where one does not: both must give the oracle's bits, and the
mixed mode must stay with it.  Cases: conductances and capacitances scaled out of the range,
a resting network (numerators of exactly zero), and trees that are one node, one chain, a star
wider than a warp and than a CTA, and a bush.
"""
import numpy as np
import pytest

import mind_b200 as mb
import oracle
from mind_b200.runtime import DeviceState

pytestmark = pytest.mark.gpu


def _sections(shape):
    soma = mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0)
    dend = lambda name, parent, nseg: mb.Section(name, label="dend", parent=parent, parent_x=1.0, length=10.0 * nseg,
                                                 diameter=2.0, nseg=nseg, Ra=100.0, cm=1.0)
    if shape == "soma":
        return [soma]
    if shape == "chain":
        return [soma, dend("d0", "soma", 70)]
    if shape == "star":
        return [soma] + [dend(f"d{k}", "soma", 1 + k % 5) for k in range(140)]
    secs = [soma, dend("d0", "soma", 3)]
    for k in range(1, 63):   # a complete binary bush with uneven branches
        secs.append(dend(f"d{k}", f"d{(k - 1) // 2}", 1 + (7 * k) % 4))
    return secs


def _layout(shape, synapses=True):
    model = mb.MicroModel(celsius=6.3)
    secs = _sections(shape)
    cells = mb.add_population(model, secs, 3, voltage=lambda k: -65.0 - 0.5 * k if synapses else -65.0)
    for cell in cells:
        if synapses:
            mb.insert(cell, mb.builtin("hh"), sections="soma")
        else:
            mb.insert(cell, mb.builtin("pas"), sections="soma", params={"g": 1e-4, "e": -65.0})
        if len(secs) > 1:
            mb.insert(cell, mb.builtin("pas"), sections="dend", params={"g": 1e-4, "e": -65.0})
        mb.register_spike_source(cell, threshold=-10.0)
    if synapses:
        for cell in cells:
            mb.add_pointprocess(cell, mb.builtin("IClamp"), params={"del": 0.5, "dur": 5.0, "amp": 0.5})
    return mb.build(model)


def _run(layout, precision, steps, nodes):
    state = DeviceState(layout, precision)
    state.initialize()
    result = state.run_steps(steps, [mb.RecordSpec(int(n), f"n{n}") for n in nodes])
    state.close()
    return result.traces.by_record.T, result


@pytest.mark.parametrize("shape", ["soma", "chain", "star", "bush"])
@pytest.mark.parametrize("change", ["none", "rest", "axial", "one axial", "capacitance"])
def test_solve_equals_the_oracle(shape, change):
    layout = _layout(shape, synapses=change != "rest")
    if change == "axial":            # below 2^-480: every axial term vanishes, every step divides
        layout.axial *= 2.0 ** -500
        layout.axial_diagonal *= 2.0 ** -500
    elif change == "one axial":
        layout.axial[-1] *= 2.0 ** -500
    elif change == "capacitance":    # pivots above 2^480
        layout.capacitance *= 2.0 ** 500
        layout.capacitance[layout.capacitance == 0.0] = 2.0 ** 500
    steps = 200
    nodes = np.unique(np.linspace(1, layout.n_nodes, 12).astype(int))
    ref = oracle.run(layout, steps, nodes)
    assert ref.status == 0, ref.message
    trace, result = _run(layout, "fp64", steps, nodes)
    assert np.array_equal(trace, ref.trace), float(np.max(np.abs(trace - ref.trace)))
    np.testing.assert_array_equal(result.spike_times, ref.spike_times)
    # mixed: FP32 gating (bound of the mixed mode's own parity tests over a spike)
    mixed, _ = _run(layout, "mixed", steps, nodes)
    assert np.max(np.abs(mixed - ref.trace)) < 0.1


def test_256_threads_per_cell_equal_64():
    """A small network runs 256 threads per cell, two on an owner slot; asked for 64 threads, two
    slots on one.  hh and pas share the soma here, in both orders, with synapses on top."""
    for first, second in (("hh", "pas"), ("pas", "hh")):
        model = mb.MicroModel(celsius=6.3)
        secs = _sections("bush")
        for k, cell in enumerate(mb.add_population(model, secs, 5, voltage=-65.0)):
            mb.insert(cell, mb.builtin(first))
            mb.insert(cell, mb.builtin(second), sections="soma" if second == "pas" else "dend")
            mb.register_spike_source(cell, threshold=-10.0)
            mb.add_pointprocess(cell, mb.builtin("IClamp"), section="d9", params={"del": 0.2, "dur": 3.0, "amp": 0.2 + 0.1 * k})
            mb.add_pointprocess(cell, mb.builtin("AlphaSynapse"), section="d9", params={"onset": 0.5, "tau": 1.0, "gmax": 0.01})
        layout = mb.build(model)
        steps = 160
        nodes = np.unique(np.linspace(1, layout.n_nodes, 15).astype(int))
        ref = oracle.run(layout, steps, nodes)
        assert ref.status == 0, ref.message
        records = [mb.RecordSpec(int(n), f"n{n}") for n in nodes]
        for threads in (128, 64):
            state = DeviceState(layout, "fp64")
            state.set_bin_threads([threads] * len(state.bin_threads()))
            state.initialize()
            trace = state.run_steps(steps, records).traces.by_record.T
            state.close()
            assert np.array_equal(trace, ref.trace), (first, threads, float(np.max(np.abs(trace - ref.trace))))
