"""A fetch allocates nothing on the device: the log is sorted with what the
context holds, by turns of steps and pieces of spikes where these are more than it
has room for at a time, and on the host where a turn holds few.  A fetch that is
refused for a small buffer takes nothing: not the spikes, not their order, not the
rows."""
import ctypes

import numpy as np
import pytest
import torch

from eden_gb300 import lowering, workloads
from eden_gb300.engine import CRecords, EdenGpuError, Simulation
from eden_gb300.network import Izhikevich2007Cell, NetworkSpec, OutputColumn, Population, SpikeArrayCell

pytestmark = pytest.mark.gpu


def _listed(n_src, steps, events, seed):
    """A neuron beside n_src spike lists, and `events` different (step, source)
    pairs of theirs in `steps` steps."""
    spec = NetworkSpec("lists", 0.1, 0.1 * steps + 1.0, 9)
    spec.cells.append(Izhikevich2007Cell("iz", a=0.03, d=10.0, c=-50.0))
    spec.populations.append(Population("p", "iz", 1))
    spec.cells.append(SpikeArrayCell("sa", np.array([0.1 * steps])))
    spec.populations.append(Population("s", "sa", n_src))
    spec.trace_columns.append(OutputColumn("p", 0, 0))
    low = lowering.lower(spec)
    rng = np.random.default_rng(seed)
    lists = np.nonzero(low.src_target < 0)[0]
    keys = rng.choice((steps - 2) * n_src, events, replace=False)
    keys.sort()
    low.ext_step = (2 + keys // n_src).astype(np.int64)
    # (sources of a step in any order)
    low.ext_src = lists[rng.permutation(n_src)[keys % n_src]].astype(np.int32)
    return low


def _check(rec, low):
    order = np.lexsort((low.ext_src, low.ext_step))
    np.testing.assert_array_equal(rec.spike_step, low.ext_step[order])
    np.testing.assert_array_equal(rec.spike_src, low.ext_src[order])
    assert np.isnan(rec.spike_time).all()


# a turn is 2^21 words of 32 sources: 1,500 steps of 100,000 sources are three;
# a piece an eighth of the log's capacity: 5,000 spikes of 40,000
@pytest.mark.parametrize("n_src,steps,events,capacity", [
    (100000, 1500, 30000, 40000),    # three turns of two pieces each
    (100000, 1500, 3073, 40000),     # just more than a thousand a turn
    (100000, 1500, 3072, 40000),     # just not: on the host
    (70, 600, 5001, 40000),          # one turn, one spike past a piece
    (70, 600, 5000, 40000),
    (31, 600, 4097, 4200),           # a small log's pieces are not smaller than 4,096
])
def test_turns_and_pieces(n_src, steps, events, capacity):
    low = _listed(n_src, steps, events, seed=events)
    sim = Simulation(low, record_capacity_steps=steps, spike_capacity=capacity)
    sim.initialize()
    sim.run_steps(steps)
    _check(sim.fetch(), low)
    sim.close()


def test_allocates_nothing():
    low = _listed(100000, 1500, 30000, seed=1)
    sim = Simulation(low, record_capacity_steps=1500)
    sim.initialize()
    sim.run_steps(1500)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    rec = sim.fetch()
    assert torch.cuda.mem_get_info(0)[0] == free
    _check(rec, low)
    sim.close()


def test_a_refused_fetch_takes_nothing():
    low = lowering.lower(workloads.izh_net(n_cells=3000, in_degree=10, length_ms=50.0))
    want, sim = (Simulation(low, record_capacity_steps=400) for _ in range(2))
    for s in (want, sim):
        s.initialize()
        s.run_steps(400)
    a = want.fetch()
    assert len(a.spike_src) > 4096   # more than the first buffer that a fetch of Simulation tries
    # the C entry, with room for the rows and one spike too few
    n = len(a.spike_src) - 1
    trace, tstep = np.zeros((400, a.trace.shape[1]), np.float32), np.zeros(400, np.int64)
    src, step = np.full(n, -7, np.int32), np.full(n, -7, np.int64)
    rec = CRecords()
    rec.trace = trace.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    rec.trace_step = tstep.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    rec.trace_capacity = 400
    rec.spike_src = src.ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
    rec.spike_step = step.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    rec.spike_capacity = n
    assert sim.lib.edenGpuFetchRecords(sim.ctx, ctypes.byref(rec)) == -5   # EDEN_GPU_E_RANGE
    assert rec.n_spikes == n + 1 and rec.n_trace_samples == 400
    assert (src == -7).all() and (step == -7).all() and not trace.any()
    sim.spike_capacity = n
    with pytest.raises(EdenGpuError):
        sim.fetch()
    sim.spike_capacity = 1 << 22
    b = sim.fetch()
    for name in ("trace", "trace_step", "spike_src", "spike_step", "spike_time"):
        np.testing.assert_array_equal(getattr(b, name), getattr(a, name))
    want.close()
    sim.close()


@pytest.mark.parametrize("n", [1, 4096, 4097])
def test_potentials_in_the_callers_order(n):
    """Few potentials are put in order on the host, many on the device: written,
    read, and written again between steps, they are the ones the next steps start
    from."""
    low = lowering.lower(workloads.single_comp_hh(n_cells=n, length_ms=5.0, n_recorded=1))
    v = np.random.default_rng(n).uniform(-75.0, -55.0, n).astype(np.float32)
    traces = []
    for target in (0, n - 1):
        sim = Simulation(low, trace_target=[target], record_capacity_steps=64)
        sim.initialize()
        np.testing.assert_array_equal(sim.read_v(), np.float32(-65.0))
        sim.write_v(v)
        w = v.copy()
        v[:] = 0.0      # the caller's array is its own again
        np.testing.assert_array_equal(sim.read_v(), w)
        sim.write_v(w)
        sim.run_steps(20)
        traces.append(sim.fetch().trace[0, 0])
        assert traces[-1] == w[target]
        assert not np.array_equal(sim.read_v(), w)
        v[:] = w
        sim.close()


def test_records_do_not_keep_the_buffers():
    """A program that fetches often and keeps the records holds what is in them."""
    low = lowering.lower(workloads.single_comp_hh(n_cells=50, length_ms=20.0, n_recorded=10))
    sim = Simulation(low, record_capacity_steps=4096)
    sim.initialize()
    sim.run_steps(7)
    rec = sim.fetch()
    sim.close()
    assert rec.trace.shape == (7, 10)
    for a in (rec.trace, rec.trace_step, rec.spike_src, rec.spike_step, rec.spike_time):
        held = a if a.base is None else a.base
        assert held.nbytes == a.nbytes
