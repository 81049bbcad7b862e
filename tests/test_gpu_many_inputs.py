"""Compartments and point neurons with many inputs of a type: their blocks are cut
into chunks of 128, whose series the cell kernel sums before the window's steps.
One chunk, two, and counts around the eight that are loaded at a time, the last
chunk part full, alone and beside blocks of one chunk; windows of lengths that are
and are not multiples of four steps.  Against the oracle by the criteria of
tests/test_gpu_parity.py (spikes within 0.1 ms, potentials inside box(0.1 ms,
0.5 mV)); the built-in kernels give the same bits as those compiled for the model."""
import numpy as np
import pytest

import eden_port
from criteria import box_violations, samecount
from eden_gb300 import lowering
from eden_gb300.engine import MODE_PLAIN, Simulation
from eden_gb300.network import (SYN_EXPONE, SYN_EXPTWO, ChannelDensity, Izhikevich2007Cell, NetworkSpec, OutputColumn,
                                PhysicalCell, PoissonInputs, Population, PulseInputs, SynapseType, hh_channels)
from helpers import spike_trains

pytestmark = pytest.mark.gpu

# inputs of the first type on each cell's first compartment; of the second, 40
COUNTS = [1, 128, 129, 255, 8 * 128, 9 * 128, 9 * 128 + 1, 17 * 128, 20 * 128 - 5, 300]


def _network(point):
    spec = NetworkSpec("many", 0.1 if point else 0.025, 40.0 if point else 12.0, 4, channels=[] if point else hh_channels())
    n = len(COUNTS)
    if point:
        spec.cells.append(Izhikevich2007Cell("c", a=0.03, d=100.0, c=-50.0))
    else:
        seg = np.ones(3, bool)
        soma = np.array([True, False, False])
        dens = [ChannelDensity(0, 0.3, -54.387, seg), ChannelDensity(1, 120.0, 50.0, soma), ChannelDensity(2, 36.0, -77.0, soma)]
        spec.cells.append(PhysicalCell("c", np.array([-1, 0, 1]), np.array([20.0, 30.0, 30.0]), np.array([20.0, 3.0, 2.0]),
                                       dens, cm=1.0, ra=150.0, spike_thresh=-20.0))
    spec.populations.append(Population("p", "c", n))
    spec.synapses.append(SynapseType("a", SYN_EXPONE, gbase=0.02, erev=0.0, tau_decay=3.0))
    spec.synapses.append(SynapseType("b", SYN_EXPTWO, gbase=0.3, erev=-70.0, tau_decay=5.0, tau_rise=0.5))
    for c, k in enumerate(COUNTS):
        spec.poissons.append(PoissonInputs("p", "a", 20.0, np.full(k, c), np.zeros(k, int)))
        spec.poissons.append(PoissonInputs("p", "b", 20.0, np.full(40, c), np.full(40, 0 if point else 2)))
    gids = np.arange(n)
    amp = np.full(n, 0.4 if point else 2.0)
    spec.pulses.append(PulseInputs("*", gids, 0 * gids, np.full(n, 1.0), np.full(n, 100.0), amp))
    spec.trace_columns = [OutputColumn("p", c, 0) for c in range(n)]
    return lowering.lower(spec)


@pytest.mark.parametrize("K", [31, 8, 5, 1])
@pytest.mark.parametrize("point", [True, False], ids=["neurons", "compartments"])
def test_blocks_of_many_chunks(point, K):
    low = _network(point)
    runs = []
    for options in (dict(), dict(codegen=-1)):
        sim = Simulation(low, steps_per_launch=K, **options)
        runs.append(sim.run())
        sim.close()
    a, b = runs
    for name in ("trace", "spike_src", "spike_step"):
        np.testing.assert_array_equal(getattr(a, name), getattr(b, name))
    ref = eden_port.run(low)
    assert len(ref["spike_src"]) > 0
    dt_ms = float(low.dt) * 1e-3
    wrong, far = samecount(spike_trains(ref["spike_src"], ref["spike_step"]), spike_trains(a.spike_src, a.spike_step),
                           int(round(0.1 / dt_ms)))
    assert not wrong and not far
    nbad, worst = box_violations(ref["trace"], a.trace, dt_ms, 0.1, 0.5)
    assert nbad == 0, f"{nbad} samples outside box(0.1 ms, 0.5 mV), worst by {worst} mV"


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_potentials_that_are_not_finite(value):
    """An input adds nothing to a sum it is not part of, whatever the potential:
    what overflows to infinity or NaN in windows is what does step by step."""
    low = _network(True)
    out = []
    for options in (dict(mode=MODE_PLAIN), dict(steps_per_launch=1)):
        sim = Simulation(low, **options)
        sim.initialize()
        sim.run_steps(100)
        v = sim.read_v()
        v[::2] = value
        sim.write_v(v)
        sim.run_steps(1)
        out.append(sim.read_v())
        sim.close()
    for f in (np.isnan, np.isposinf, np.isneginf):
        np.testing.assert_array_equal(f(out[0]), f(out[1]))
    assert np.isfinite(out[0][1::2]).all()
