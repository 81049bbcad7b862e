"""How the windowed kernel packs cells into units changes no compartment's
operations: whatever the packing -- which decides the subtrees a lane walks by
itself, the passes above them and the warps of a block -- every potential is the
same bit for bit.  Trees where that can go wrong: a star with more children than
a warp has lanes, a chain, a random tree, a cell of one compartment, and active
compartments far from the soma."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import Simulation
from eden_gb300.network import ChannelDensity, NetworkSpec, OutputColumn, PhysicalCell, Population, PulseInputs, hh_channels

pytestmark = pytest.mark.gpu


def _trees():
    rng = np.random.default_rng(3)
    star = np.concatenate([[-1], np.zeros(70, np.int64)])
    brooms = np.concatenate([[-1], np.arange(8), np.full(40, 8)])
    trees = [np.array([-1]), star, np.arange(-1, 89), brooms]
    trees += [workloads.random_tree(rng, n)[0] for n in (2, 31, 33, 300)]
    spec = NetworkSpec("packing", 0.025, 5.0, 7, channels=hh_channels())
    for k, parent in enumerate(trees):
        n = len(parent)
        hh = rng.random(n) < (0.2 if k % 2 else 0.0)
        hh[0] = True
        dens = [ChannelDensity(0, 0.3, -54.387, np.ones(n, bool)), ChannelDensity(1, 120.0, 50.0, hh),
                ChannelDensity(2, 36.0, -77.0, hh)]
        length, diam = rng.uniform(5.0, 50.0, n), rng.uniform(0.5, 4.0, n)
        length[0] = diam[0] = 20.0
        spec.cells.append(PhysicalCell(f"c{k}", parent, length, diam, dens, cm=1.0, ra=150.0))
        spec.populations.append(Population(f"p{k}", f"c{k}", 3))
        spec.trace_columns += [OutputColumn(f"p{k}", 1, s) for s in sorted({0, n // 2, n - 1})]
    cells = np.arange(3 * len(trees))
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(len(cells)), np.full(len(cells), 5.0),
                                   rng.uniform(0.1, 0.6, len(cells))))
    return lowering.lower(spec)


@pytest.fixture(scope="module")
def default():
    low = _trees()
    sim = Simulation(low)
    rec = sim.run(150)
    v = sim.read_v()
    sim.close()
    return low, rec.trace, v


@pytest.mark.parametrize("packing", [dict(segments_per_warp=8), dict(segments_per_warp=64), dict(segments_per_warp=1023),
                                     dict(segments_per_warp=1023, segments_per_depth=1023),
                                     dict(segments_per_warp=1023, segments_per_depth=4), dict(max_cell_blocks=1),
                                     dict(codegen=-1)], ids=str)
def test_packing_changes_no_potential(packing, default):
    low, trace, v = default
    sim = Simulation(low, **packing)
    rec = sim.run(150)
    np.testing.assert_array_equal(rec.trace, trace)
    np.testing.assert_array_equal(sim.read_v(), v)
    sim.close()
