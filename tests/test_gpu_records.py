"""Fetched spikes come in order of step, then source, whatever the log's size:
sorted on the host up to a thousand or so, by counting bits on the device above,
and on the host again where a source is listed twice in a step.  Each case is
compared with the same run fetched in pieces of whole windows (10 steps: cutting a
window short would round its synapses' closed forms differently); potentials
written and read back are the same."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import EdenGpuError, Simulation

pytestmark = pytest.mark.gpu


def _pairs(rec):
    return np.stack([rec.spike_step, rec.spike_src.astype(np.int64)], 1)


def _is_sorted(p):
    d = np.diff(p, axis=0)
    return bool(((d[:, 0] > 0) | ((d[:, 0] == 0) & (d[:, 1] >= 0))).all())


@pytest.mark.parametrize("n_cells,steps", [(33, 2000), (2000, 400), (5000, 1000)])
def test_order_and_content(n_cells, steps):
    low = lowering.lower(workloads.izh_net(n_cells=n_cells, in_degree=10, length_ms=200.0))
    whole = Simulation(low, record_capacity_steps=steps)
    a = whole.run(steps)
    pieces = Simulation(low, record_capacity_steps=steps)
    b = pieces.run(steps, chunk=20)
    np.testing.assert_array_equal(whole.read_v(), pieces.read_v())
    whole.close()
    pieces.close()
    assert len(a.spike_src) > n_cells and _is_sorted(_pairs(a))
    np.testing.assert_array_equal(_pairs(a), _pairs(b))


def test_a_source_listed_twice_in_a_step():
    low = lowering.lower(workloads.spike_sources(length_ms=50.0))
    src = int(np.nonzero(low.src_target < 0)[0][0])
    # 1,500 entries in 30 steps, every one there twice or more
    low.ext_step = np.repeat(np.arange(2, 32), 50).astype(np.int64)
    low.ext_src = np.full(len(low.ext_step), src, np.int32)
    sim = Simulation(low, record_capacity_steps=64)
    rec = sim.run(40)
    sim.close()
    p = _pairs(rec)
    assert _is_sorted(p) and (p[:, 1] == src).sum() == 1500


def test_too_small_a_buffer_takes_nothing():
    low = lowering.lower(workloads.izh_net(n_cells=500, in_degree=10, length_ms=50.0))
    sim = Simulation(low, record_capacity_steps=400)
    sim.initialize()
    sim.run_steps(300)
    # the same log twice as large as the first buffer the fetch tries
    rec = sim.fetch()
    assert len(rec.trace_step) == 300 and rec.trace_step[0] == 1
    sim.run_steps(100)
    sim.record_capacity_steps = 50
    with pytest.raises(EdenGpuError):
        sim.fetch()
    sim.record_capacity_steps = 400
    rec = sim.fetch()
    assert len(rec.trace_step) == 100 and rec.trace_step[0] == 301
    sim.close()


def test_potentials_round_trip():
    low = lowering.lower(workloads.multicomp_net(n_cells=20, in_degree=5, length_ms=5.0, max_seg=60))
    sim = Simulation(low)
    v = np.linspace(-80.0, -50.0, low.n_target).astype(np.float32)
    sim.write_v(v)
    np.testing.assert_array_equal(sim.read_v(), v)
    sim.close()
