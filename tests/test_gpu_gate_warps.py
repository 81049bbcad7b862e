"""Units whose gates have a warp of their own compute the same bits as units of
one warp: 20,000 HH cells in units of 8 are too many for two warps each to be
resident, in the default's they are not; more than 32 compartments and gates a
unit, more CTAs than blocks, the built-in kernels, and units without a gate
beside units with."""
import numpy as np
import pytest

from eden_gb300 import lowering
from eden_gb300.engine import Simulation
from eden_gb300.network import ChannelDensity, NetworkSpec, OutputColumn, PhysicalCell, Population, PulseInputs, hh_channels

pytestmark = pytest.mark.gpu


def _network(passive):
    rng = np.random.default_rng(5)
    spec = NetworkSpec("gate warps", 0.025, 5.0, 3, channels=hh_channels())
    one, all_ = np.array([-1]), np.ones(1, bool)
    leak = ChannelDensity(0, 0.3, -54.387, all_)
    hh = [leak, ChannelDensity(1, 120.0, 50.0, all_), ChannelDensity(2, 36.0, -77.0, all_)]
    spec.cells.append(PhysicalCell("hh", one, np.full(1, 17.8), np.full(1, 17.8), hh, cm=1.0, ra=30.0, spike_thresh=-20.0))
    spec.cells.append(PhysicalCell("leak", one, np.full(1, 17.8), np.full(1, 17.8), [leak], cm=1.0, ra=30.0))
    n = 2000 if passive else 20000
    spec.populations.append(Population("a", "hh", n))
    if passive:
        spec.populations.append(Population("b", "leak", passive))
    cells = np.arange(n + passive)
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, rng.uniform(0, 2, len(cells)), np.full(len(cells), 4.0),
                                   rng.uniform(0.05, 0.3, len(cells))))
    spec.trace_columns += [OutputColumn("a", int(c), 0) for c in range(0, n, 97)]
    spec.trace_columns += [OutputColumn("b", int(c), 0) for c in range(0, passive, 97)]
    return lowering.lower(spec)


def _run(low, **options):
    sim = Simulation(low, **options)
    rec = sim.run()
    v = sim.read_v()
    sim.close()
    return rec.trace, rec.spike_src, rec.spike_step, v


@pytest.fixture(scope="module")
def one_warp():
    cache = {}

    def get(passive):
        if passive not in cache:
            low = _network(passive)
            cache[passive] = (low, _run(low, segments_per_warp=8))
        return cache[passive]
    return get


@pytest.mark.parametrize("options", [dict(), dict(segments_per_warp=32), dict(segments_per_warp=33), dict(segments_per_warp=100),
                                     dict(max_cell_blocks=1), dict(codegen=-1), dict(steps_per_launch=7)], ids=str)
@pytest.mark.parametrize("passive", [0, 18000])
def test_two_warps_compute_the_same(passive, options, one_warp):
    low, want = one_warp(passive)
    assert len(want[1]) > 1000
    for a, b in zip(_run(low, **options), want):
        np.testing.assert_array_equal(a, b)
