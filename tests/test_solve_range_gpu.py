"""Networks at the limits of the range in which the FP64 solve forms its quotients by FMA, and across
them, against the oracle: bit-identical wherever a step is solved with the quotients, solved again
with divisions, or divided at once because the step before it was.

Cases: a cable at rest whose change from a stimulus fades to nothing along the way (from the first
step, from a pulse in mid-run, and in calls of few steps, between which a cell keeps whether it
divides), one that fades within the range, the whole system scaled to just inside the limits, and one cell
of three outside them.
"""
import numpy as np
import pytest

import mind_b200 as mb
import oracle
from mind_b200.runtime import DeviceState

pytestmark = pytest.mark.gpu


def _cable(nseg, cells=2, delay=0.0):
    model = mb.MicroModel(celsius=6.3)
    secs = [mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0),
            mb.Section("d", label="dend", parent="soma", parent_x=1.0, length=50.0 * nseg, diameter=0.5, nseg=nseg,
                       Ra=100.0, cm=1.0)]
    for cell in mb.add_population(model, secs, cells, voltage=-65.0):
        mb.insert(cell, mb.builtin("pas"), params={"g": 1e-4, "e": -65.0})
        mb.add_pointprocess(cell, mb.builtin("IClamp"), params={"del": delay, "dur": 0.5, "amp": 0.1})
    return mb.build(model)


def _scale(layout, power):
    layout.axial *= 2.0 ** power
    layout.axial_diagonal *= 2.0 ** power
    layout.capacitance *= 2.0 ** power


CASES = {
    "fades in range": (lambda: _cable(90), None),
    "fades to nothing": (lambda: _cable(700), None),
    "from a pulse": (lambda: _cable(700, delay=0.8), None),
    "scaled up": (lambda: _cable(60), lambda l: _scale(l, 470)),
    "scaled down": (lambda: _cable(60), lambda l: _scale(l, -470)),
    "one cell of three": (lambda: _cable(60, cells=3), lambda l: l.axial.__setitem__(l.n_nodes // 2, 2.0 ** -490)),
}


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("call", [120, 7])
def test_solve_across_its_range(case, call):
    make, change = CASES[case]
    layout = make()
    if change:
        change(layout)
    steps = 120
    nodes = np.unique(np.linspace(1, layout.n_nodes, 24).astype(int))
    ref = oracle.run(layout, steps, nodes)
    assert ref.status == 0, ref.message
    records = [mb.RecordSpec(int(n), f"n{n}") for n in nodes]
    state = DeviceState(layout, "fp64")
    for _ in range(2):
        state.initialize()
        for first in range(0, steps, call):
            n = min(call, steps - first)
            trace = state.run_steps(n, records).traces.by_record.T
            assert np.array_equal(trace, ref.trace[first:first + n + 1]), (first, float(np.max(np.abs(
                trace - ref.trace[first:first + n + 1]))))
    state.close()
