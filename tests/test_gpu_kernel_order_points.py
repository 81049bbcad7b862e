"""Networks of point neurons alone, step by step: they have no forest, so the
kernel of the cable solves has nothing to do, and must still keep its place
between the neurons' kernel and the delivery.  With synapses between them a lost
spike, or one delivered twice, shows in what follows.  Timing each kernel puts
events between the kernels, which order them completely; the records of the runs
without are the same bits."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import MODE_PLAIN, Simulation

pytestmark = pytest.mark.gpu


def _run(low, pieces, **options):
    sim = Simulation(low, **options)
    sim.initialize()
    out = []
    for n in pieces:
        sim.run_steps(n)
        # inputs, neurons, delivery: nothing is launched for the cables that are not there
        assert sim.last_launches == 3 * n
        rec = sim.fetch()
        out += [rec.spike_src, rec.spike_step, rec.trace, sim.read_v()]
    sim.close()
    return out


@pytest.mark.parametrize("n_cells,in_degree", [(40, 10), (3000, 50), (60000, 20)])
def test_point_neurons_step_by_step(n_cells, in_degree):
    low = lowering.lower(workloads.izh_net(n_cells=n_cells, in_degree=in_degree, length_ms=30.0, n_recorded=4))
    pieces = [150, 1, 49, 100]
    want = _run(low, pieces, mode=MODE_PLAIN, kernel_timing=True)
    assert sum(len(a) for a in want[::4]) > 0
    for _ in range(3):
        for a, b in zip(_run(low, pieces, mode=MODE_PLAIN), want):
            np.testing.assert_array_equal(a, b)
