"""Recorded mechanism state at every step, against the oracle: the record holds the state that the
step has just advanced, whichever warp advances it.

Cells of one hh row and of an hh row per node, more Exp2Syn rows than a warp records, and the
same mechanisms emitted from MOD files, whose state lies in HBM; cells of fewer nodes than a
CTA's threads and of more.
"""
import numpy as np
import pytest

import mind_b200 as mb
import oracle
from mind_b200.runtime import DeviceState

pytestmark = pytest.mark.gpu

SYNAPSES = 40


def _model(nseg, get):
    model = mb.MicroModel(celsius=6.3)
    secs = [mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0),
            mb.Section("d", label="dend", parent="soma", parent_x=1.0, length=5.0 * nseg, diameter=2.0, nseg=nseg,
                       Ra=100.0, cm=1.0)]
    cells = mb.add_population(model, secs, 2, voltage=-65.0)
    mb.insert(cells[0], get("hh"), sections="soma")
    mb.insert(cells[0], get("pas"), sections="dend", params={"g": 1e-4, "e": -65.0})
    mb.insert(cells[1], get("hh"))
    for cell in cells:
        mb.register_spike_source(cell, threshold=-10.0)
    owners = np.repeat([1, 2], SYNAPSES)
    n = len(owners)
    first = mb.add_pointprocesses(model, get("Exp2Syn"), owners, "d", np.linspace(0.02, 0.98, n),
                                  {"tau1": 0.5, "tau2": 5.0, "e": 0.0})
    stims = mb.add_pointprocesses(model, mb.builtin("NetStim"), np.zeros(n, np.int64), "none", np.zeros(n),
                                  {"interval": 2.0, "number": 1e9, "start": 0.0, "noise": 1.0})
    sources = mb.register_point_sources(model, np.arange(stims, stims + n))
    mb.connect_many(model, sources, np.arange(first, first + n), np.full(n, 4e-4), np.zeros(n))
    return model


@pytest.mark.parametrize("emitted", [False, True])
@pytest.mark.parametrize("nseg", [70, 140])
def test_recorded_state_is_the_step_s(nseg, emitted):
    model = _model(nseg, mb.emitted if emitted else mb.builtin)
    layout = mb.build(model)
    hh_rows = [g for g in layout.groups if g.mechanism.name == "hh"][0].rows
    recs = [mb.RecordSpec(layout.voltage_node(c), f"v{c}") for c in (1, 2)]
    recs += [mb.mechanism_ref(model, "hh", r, f) for r in sorted({1, 2, hh_rows // 2, hh_rows}) for f in ("m", "h", "n")]
    recs += [mb.mechanism_ref(model, "Exp2Syn", r, f) for r in range(1, 2 * SYNAPSES + 1) for f in ("A", "B")]
    steps = 600
    ref = oracle.run(layout, steps, records=recs)
    assert ref.status == 0, ref.message
    for threads in (None,) if emitted else (None, 64, 32):   # None: the shape the library chooses
        state = DeviceState(layout, "fp64")
        if threads:
            state.set_bin_threads([threads] * len(state.bin_threads()))
        for _ in range(3):
            state.initialize()
            trace = state.run_steps(steps, recs).traces.by_record.T
            assert np.array_equal(trace, ref.trace), (threads, float(np.max(np.abs(trace - ref.trace))))
        state.close()
    assert ref.trace[:, -1].max() > 0.0   # events arrived
