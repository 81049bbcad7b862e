"""Spikes of point neurons taken into a window's list together, and a window's
spikes logged 32 at a time, at the sizes where they can go wrong: every neuron of
a warp spiking in one step, neurons that spike several times in a window (every 6
of its 31 steps), the last warp part full, more spikes than the delivery's warps log in one pass, and
spikes of sources without a target beside them.  One-step windows log every step
by itself: the spikes are the same ones."""
import numpy as np
import pytest

from eden_gb300 import lowering
from eden_gb300.engine import MODE_BATCHED, MODE_PLAIN, Simulation
from eden_gb300.network import (Izhikevich2007Cell, NetworkSpec, OutputColumn, Population, PulseInputs, SpikeArrayCell)

pytestmark = pytest.mark.gpu


def _network(n, arrays, d, amplitude):
    spec = NetworkSpec("spikes", 0.1, 40.0, 9)
    # every neuron the same and driven the same: all spike in the same steps
    spec.cells.append(Izhikevich2007Cell("iz", a=0.03, d=d, c=-50.0))
    spec.populations.append(Population("p", "iz", n))
    if arrays:
        spec.cells.append(SpikeArrayCell("sa", np.arange(1.0, 39.0, 0.3)))
        spec.populations.append(Population("s", "sa", arrays))
    cells = np.arange(n)
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(n), np.full(n, 40.0), np.full(n, amplitude)))
    spec.trace_columns.append(OutputColumn("p", n - 1, 0))
    return lowering.lower(spec)


@pytest.mark.parametrize("d,amplitude,spikes", [(10.0, 2.0, 13), (0.0, 20.0, 66)])
@pytest.mark.parametrize("n,arrays", [(1, 0), (31, 2), (33, 0), (1000, 40), (160001, 3)])
def test_windows_list_the_spikes_of_their_steps(n, arrays, d, amplitude, spikes):
    low = _network(n, arrays, d, amplitude)
    runs = []
    for options in (dict(steps_per_launch=1), dict(mode=MODE_PLAIN), dict(), dict(codegen=-1), dict(steps_per_launch=31)):
        sim = Simulation(low, **options)
        rec = sim.run(chunk=31)
        runs.append((rec.spike_src, rec.spike_step, rec.trace))
        sim.close()
    own = runs[0][0] < n
    counts = np.bincount(runs[0][0][own], minlength=n)
    assert counts.min() == counts.max() == spikes
    for run in runs[1:]:
        for a, b in zip(run, runs[0]):
            np.testing.assert_array_equal(a, b)
