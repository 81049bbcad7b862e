"""The input kernel at the sizes where it can go wrong: blocks of one item, of
rows of 32 just filled and just passed, of a chunk of 128 just filled and just
passed, more items with an event in a window than the list of a group of chunks
holds, items that fire more than once in a window, and several kinds and
synapse types side by side.

Tolerance: a step rounds a potential below 128 mV to 2^-17 mV and its few
terms by as much, so 400 steps stay within 400 * 4 * 2^-17 = 0.012 mV of the
oracle's even where nothing decays.  One event lost or doubled moves it by more:
0.04 mV (e1: 0.01 nS for 2 ms at 60 mV into 28 pF), 0.02 mV (e2: 3 ms at 20 mV)."""
import numpy as np
import pytest

import eden_port
from eden_gb300 import lowering
from eden_gb300.engine import MODE_BATCHED, MODE_PLAIN, Simulation
from eden_gb300.network import (SYN_ALPHA, SYN_EXPONE, SYN_EXPTWO, ChannelDensity, NetworkSpec, OutputColumn, PhysicalCell,
                                PoissonInputs, Population, Projection, PulseInputs, SpikeGeneratorCell, SynapseType,
                                TimedInputs, hh_channels)

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 64, 97, 127, 128, 129, 257]
COPIES = 130  # enough chunks for groups of several on every warp
STEPS = 400


def _network(kinds):
    rng = np.random.default_rng(11)
    size = np.tile(SIZES, COPIES)
    nc = len(size)
    spec = NetworkSpec("inputs", 0.025, STEPS * 0.025, 5, channels=hh_channels())
    one = np.array([-1])
    spec.cells.append(PhysicalCell("c", one, np.full(1, 30.0), np.full(1, 30.0),
                                   [ChannelDensity(0, 0.3, -60.0, np.ones(1, bool))], cm=1.0, ra=150.0))
    spec.populations.append(Population("p", "c", nc))
    # many targets' synapses of one source have their event in the same step
    for k, period in enumerate((0.4, 2.3)):
        spec.cells.append(SpikeGeneratorCell(f"g{k}", period))
        spec.populations.append(Population(f"s{k}", f"g{k}", 3))
    spec.synapses += [SynapseType("e1", SYN_EXPONE, 0.01, 0.0, 2.0), SynapseType("e2", SYN_EXPTWO, 0.01, -80.0, 3.0, 0.5),
                      SynapseType("al", SYN_ALPHA, 0.01, 0.0, 1.0)]
    cell = np.repeat(np.arange(nc), size)
    n = len(cell)
    for name in kinds:
        if name == "pulse":
            spec.pulses.append(PulseInputs("*", cell, 0 * cell, rng.uniform(0, 5, n), rng.uniform(0, 5, n),
                                           rng.uniform(0, 2e-4, n)))
        elif name == "timed":
            times = [np.sort(rng.uniform(0, 10, rng.integers(0, 12))) for _ in range(n)]
            spec.timed.append(TimedInputs("e2", cell, 0 * cell, times, rng.uniform(0.5, 1.5, n)))
        elif name.startswith("pois"):
            # intervals of a few steps: several firings in a window
            spec.poissons.append(PoissonInputs("*", name[5:], 900.0, cell[::2], 0 * cell[::2]))
        else:
            for k in range(2):
                part = cell[k::2]
                spec.projections.append(Projection(f"{name}{k}", f"s{k}", "p", name,
                                                   nc + 3 * k + rng.integers(0, 3, len(part)), part, 0 * part,
                                                   rng.uniform(0.5, 1.5, len(part)),
                                                   rng.choice([0.5, 0.725, 1.3, 3.1], len(part))))
    spec.trace_columns += [OutputColumn("p", int(c), 0) for c in range(0, nc, 7)]
    return lowering.lower(spec)


KINDS = {"synapses": ["e1", "e2"], "poisson": ["pois_e1", "pois_e2"], "one_kind": ["e1"],
         "all": ["pulse", "timed", "pois_e2", "e1", "al"]}


@pytest.fixture(scope="module")
def oracle_runs():
    cache = {}

    def get(name):
        if name not in cache:
            low = _network(KINDS[name])
            cache[name] = (low, eden_port.run(low)["trace"])
        return cache[name]
    return get


@pytest.mark.parametrize("options", [dict(), dict(codegen=-1), dict(mode=MODE_PLAIN), dict(steps_per_launch=1)], ids=str)
@pytest.mark.parametrize("kinds", list(KINDS))
def test_input_blocks_of_every_size(kinds, options, oracle_runs):
    low, trace = oracle_runs(kinds)
    sim = Simulation(low, **options)
    rec = sim.run()
    sim.close()
    assert rec.trace.shape == trace.shape
    assert np.ptp(trace, axis=0).max() > 1.0
    np.testing.assert_allclose(rec.trace, trace, rtol=0, atol=0.012)
