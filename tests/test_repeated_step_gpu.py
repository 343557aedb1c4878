"""A step whose system is solved a second time, with divisions, runs an emitted BREAKPOINT no more
often than any other step: twice, at v + 0.001 and at v.

tests/mod/UserCounter.mod counts its evaluations and sums its charge over them.  Capacitances
scaled by 2^500 put every pivot beyond the range of the quotients by FMA.
"""
import os

import numpy as np
import pytest

import mind_b200 as mb
from mind_b200.runtime import DeviceState

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("nseg", [1, 200])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 500])
def test_breakpoint_runs_twice_per_step(nseg, scale):
    counter = mb.load_mod(os.path.join(HERE, "mod", "UserCounter.mod"))
    model = mb.MicroModel(celsius=6.3)
    secs = [mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0),
            mb.Section("d", label="dend", parent="soma", parent_x=1.0, length=10.0 * nseg, diameter=2.0, nseg=nseg,
                       Ra=100.0, cm=1.0)]
    for cell in mb.add_population(model, secs, 2, voltage=-65.0):
        mb.insert(cell, mb.builtin("pas"), params={"g": 1e-4, "e": -65.0})
        for section in ("soma", "d"):
            mb.add_pointprocess(cell, counter, section=section)
    layout = mb.build(model)
    layout.capacitance *= scale
    layout.capacitance[layout.capacitance == 0.0] = scale
    nodes = [g for g in layout.groups if g.mechanism.name == "UserCounter"][0].nodes
    recs = [mb.RecordSpec(int(node), f"v{k}") for k, node in enumerate(nodes)]
    refs = [[mb.mechanism_ref(model, "UserCounter", r, f) for r in range(1, len(nodes) + 1)] for f in ("n", "q")]
    steps = 60
    state = DeviceState(layout, "fp64")
    for run in range(3):     # from rest each time: what a run keeps does not reach the next
        state.initialize()
        trace = state.run_steps(steps, recs + refs[0] + refs[1]).traces.by_record
        v, n, q = np.split(trace, 3)
        assert np.array_equal(n, np.tile(2.0 * np.arange(steps + 1), (len(nodes), 1))), n[:, -1]
        want = np.zeros(len(nodes))
        for k in range(steps):
            want = want + 0.002 * ((v[:, k] + 0.001) - -60.0) * layout.dt
            want = want + 0.002 * (v[:, k] - -60.0) * layout.dt
            assert np.array_equal(q[:, k + 1], want)
    state.close()
