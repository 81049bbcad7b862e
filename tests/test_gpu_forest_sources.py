"""The per-step kernels find a forest's spikes from its list of sources: one, 32
and more a forest, sources at the roots of trees, and forests larger than what a
warp stages, must all give the spikes and potentials of the default's forests."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import MODE_PLAIN, Simulation
from eden_gb300.network import ChannelDensity, NetworkSpec, OutputColumn, PhysicalCell, Population, PulseInputs, hh_channels

pytestmark = pytest.mark.gpu


def _network():
    rng = np.random.default_rng(8)
    spec = NetworkSpec("sources", 0.025, 8.0, 3, channels=hh_channels())
    sizes = {"one": (1, 150), "leak": (1, 40), "tree": (60, 40)}
    for name, (n, count) in sizes.items():
        parent = workloads.random_tree(rng, n)[0] if n > 1 else np.array([-1])
        soma = np.zeros(n, bool)
        soma[0] = name != "leak"
        dens = [ChannelDensity(0, 0.3, -54.387, np.ones(n, bool)), ChannelDensity(1, 120.0, 50.0, soma),
                ChannelDensity(2, 36.0, -77.0, soma)]
        length, diam = rng.uniform(5.0, 30.0, n), rng.uniform(0.5, 2.0, n)
        length[0] = diam[0] = 20.0
        spec.cells.append(PhysicalCell(name, parent, length, diam, dens, cm=1.0, ra=150.0,
                                       spike_thresh=-20.0))
        spec.populations.append(Population(f"p_{name}", name, count))
    cells = np.arange(sum(c for _, c in sizes.values()))
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, rng.uniform(0, 1, len(cells)), np.full(len(cells), 7.0),
                                   rng.uniform(0.3, 1.0, len(cells))))
    spec.trace_columns += [OutputColumn("p_tree", c, 0) for c in range(0, 40, 9)]
    return lowering.lower(spec)


def _run(low, **options):
    sim = Simulation(low, mode=MODE_PLAIN, **options)
    rec = sim.run()
    v = sim.read_v()
    sim.close()
    return rec.trace, rec.spike_src, rec.spike_step, v


@pytest.mark.parametrize("segments", [1, 32, 33, 100, 1023])
def test_forests_of_many_sources(segments):
    low = _network()
    want = _run(low)
    assert len(np.unique(want[1])) > 150
    for a, b in zip(_run(low, segments_per_warp=segments, segments_per_depth=1023), want):
        np.testing.assert_array_equal(a, b)
