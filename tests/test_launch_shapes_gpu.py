"""Launch shapes: a bin that was set to 256, 128, 64 or 32 threads per cell runs exactly those, and
says so; one at its default says 128 and launches 256 where few cells of more than 128 nodes leave
room for them.  Results do not depend on the shape, nor on when it changes.
"""
import numpy as np
import pytest

import mind_b200 as mb
import oracle
from mind_b200 import surrogate
from mind_b200.macro import MacroModel
from mind_b200.runtime import DeviceState

pytestmark = pytest.mark.gpu


def _model(cells, nseg, clamps=False, get=mb.builtin):
    model = mb.MicroModel(celsius=6.3)
    secs = [mb.Section("soma", label="soma", length=20.0, diameter=20.0, nseg=1, Ra=100.0, cm=1.0)]
    for k in range(5):
        secs.append(mb.Section(f"d{k}", label="dend", parent="soma" if k < 2 else f"d{k - 2}", parent_x=1.0,
                               length=5.0 * nseg / 5, diameter=2.0, nseg=nseg // 5, Ra=100.0, cm=1.0))
    for k, cell in enumerate(mb.add_population(model, secs, cells, voltage=lambda i: -65.0 - 0.1 * (i % 7))):
        mb.insert(cell, get("hh"), sections="soma")
        mb.insert(cell, get("pas"), sections="dend", params={"g": 1e-4, "e": -65.0})
        mb.register_spike_source(cell, threshold=-10.0)
    owners = np.arange(1, cells + 1)
    mb.add_pointprocesses(model, mb.builtin("IClamp"), owners, "d3", np.full(cells, 0.3),
                          {"del": 0.2, "dur": 4.0, "amp": 0.2 + 0.02 * (owners % 5)})
    mb.add_pointprocesses(model, get("AlphaSynapse"), owners, "d3", np.full(cells, 0.3),
                          {"onset": 0.5, "tau": 1.0, "gmax": 0.01})
    if clamps:
        mb.add_pointprocesses(model, mb.emitted("SEClamp"), owners[:2], "soma", np.full(2, 0.5),
                              {"rs": 1.0, "dur1": 1.0, "amp1": -65.0, "dur2": 1.0e9, "amp2": -50.0})
    return model


def _trace(layout, nodes, threads, precision, steps):
    state = DeviceState(layout, precision)
    if threads:
        state.set_bin_threads([threads] * len(state.bin_threads()))
    shape = state.bin_threads()
    state.initialize()
    trace = state.run_steps(steps, [mb.RecordSpec(int(n), f"n{n}") for n in nodes]).traces.by_record.T
    state.close()
    return trace, shape


@pytest.mark.parametrize("kind", ["plain", "clamps", "emitted"])
def test_every_shape_gives_the_oracle_s_bits(kind):
    layout = mb.build(_model(5, 200, kind == "clamps", mb.emitted if kind == "emitted" else mb.builtin))
    nodes = np.unique(np.linspace(1, layout.n_nodes, 17).astype(int))
    steps = 240
    ref = oracle.run(layout, steps, nodes)
    assert ref.status == 0, ref.message
    shapes = (None, 256, 128, 64, 32) if kind == "plain" else (None, 256, 128)
    mixed = []
    for threads in shapes:
        trace, shape = _trace(layout, nodes, threads, "fp64", steps)
        assert shape == [threads or 128]
        assert np.array_equal(trace, ref.trace), (threads, float(np.max(np.abs(trace - ref.trace))))
        mixed.append(_trace(layout, nodes, threads, "mixed", steps)[0])
        assert np.array_equal(mixed[-1], mixed[0]), threads
    state = DeviceState(layout, "fp64")
    for refused in (96, 512) if kind == "plain" else (64, 32):
        with pytest.raises(mb.abi.MindError):
            state.set_bin_threads([refused])
    assert state.bin_threads() == [128]      # a refused shape changes nothing
    state.close()


def test_shapes_as_the_detailed_cells_change():
    cells = 320
    model = _model(cells, 200)
    macro = MacroModel(dt_macro=0.1, bin_ms=1.0)
    region = macro.add_region(micro_gain=1.0)
    macro.add_outputs(region, list(range(1, cells + 1)))
    model.macro = macro
    layout = mb.build(model)
    net = surrogate.Mlp(seed=3)
    some = np.ones(cells, dtype=bool)
    some[:20] = False
    nodes = [layout.voltage_node(c) for c in range(1, 21)]
    recs = [mb.RecordSpec(n, f"n{n}") for n in nodes]
    runs = []
    for threads in (None, 256, 128, 64):   # by default 256 with the surrogate, 128 without it
        state = DeviceState(layout, "mixed")
        state.attach_macro(macro)
        if threads:
            state.set_bin_threads([threads] * len(state.bin_threads()))
        state.attach_surrogate(net, some, 1.0)
        state.initialize()
        parts = []
        for mask in (some, np.zeros(cells, dtype=bool), some):
            state.set_surrogate_cells(mask)
            parts.append(state.run_steps(80, recs).traces.by_record)
        assert set(state.bin_threads()) == {threads or 128}
        runs.append(np.concatenate(parts, axis=1))
        state.close()
    net.close()
    assert all(np.array_equal(r, runs[0]) for r in runs[1:])


def test_autotune_where_256_is_the_default():
    model = _model(4, 200)
    layout = mb.build(model)
    mb.initialize(model)
    shapes = mb.autotune(model, windows=2)
    assert len(shapes) == 1 and shapes[0] in (128, 64, 32)
    nodes = np.unique(np.linspace(1, layout.n_nodes, 9).astype(int))
    ref = oracle.run(layout, 120, nodes)
    got = mb.run(model, 120 * layout.dt, records=[mb.RecordSpec(int(n), f"n{n}") for n in nodes])
    assert np.array_equal(got.traces.by_record.T, ref.trace)
