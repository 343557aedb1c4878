"""More cells than the GPU has places for, of images of which another fits a multiprocessor when the hh
parameters are read from HBM: the run, with recorded hh fields, equals the oracle's, also
beside a mechanism emitted from a MOD file.

A cell of 1,120 nodes with hh on each takes about 125 KB, one to a multiprocessor of 228 KB; 63 KB
without the parameters.  150 cells exceed 148 places.
"""
import numpy as np
import pytest

import mind_b200 as mb
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clamps", [False, True])
def test_streamed_hh_parameters(clamps):
    model = mb.MicroModel(celsius=6.3)
    secs = [mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0)]
    for k in range(28):
        secs.append(mb.Section(f"d{k}", label="dend", parent="soma" if k < 4 else f"d{k - 4}", parent_x=1.0, length=300.0,
                               diameter=2.0, nseg=40, Ra=100.0, cm=1.0))
    cells = 150
    rng = np.random.default_rng(5)
    for cell in mb.add_population(model, secs, cells, voltage=lambda i: -65.0 - 0.05 * (i % 11)):
        # a parameter set of each cell's own
        mb.insert(cell, mb.builtin("hh"), params={"gnabar": float(rng.uniform(0.1, 0.14)), "el": float(rng.uniform(-56, -53))})
        mb.register_spike_source(cell, threshold=-10.0)
    owners = np.arange(1, cells + 1)
    mb.add_pointprocesses(model, mb.builtin("IClamp"), owners, "d3", np.full(cells, 0.3),
                          {"del": 0.1, "dur": 4.0, "amp": 1.0 + 0.1 * (owners % 5)})
    if clamps:
        mb.add_pointprocesses(model, mb.emitted("SEClamp"), owners[:3], "soma", np.full(3, 0.5),
                              {"rs": 1.0, "dur1": 0.5, "amp1": -65.0, "dur2": 1.0e9, "amp2": -50.0})
    layout = mb.build(model)
    rows = [g for g in layout.groups if g.mechanism.name == "hh"][0].rows
    recs = [mb.RecordSpec(int(n), f"n{n}") for n in np.linspace(1, layout.n_nodes, 60).astype(int)]
    recs += [mb.mechanism_ref(model, "hh", int(r), f) for r in np.linspace(1, rows, 20).astype(int)
             for f in ("m", "h", "n", "gnabar", "el")]
    steps = 50
    ref = oracle.run(layout, steps, records=recs)
    assert ref.status == 0, ref.message
    for precision in ("fp64", "mixed"):
        mb.initialize(model, precision=precision)
        trace = mb.run(model, steps * layout.dt, records=recs).traces.by_record.T
        if precision == "fp64":
            assert np.array_equal(trace, ref.trace), float(np.max(np.abs(trace - ref.trace)))
        else:                # FP32 gating: the bound of the mixed mode's own parity tests
            assert np.max(np.abs(trace - ref.trace)) < 0.1
