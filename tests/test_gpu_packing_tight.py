"""Units that only just fit the SMs' shared memory in one round -- 10,000 trees fill
98 % of it and need exchanges between the blocks to be placed -- and networks on
either side of it, compute the same bits as packed otherwise, whether or not a
window's kernels start early."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import Simulation

pytestmark = pytest.mark.gpu


def _run(low, **options):
    sim = Simulation(low, **options)
    sim.initialize()
    sim.run_steps(120)
    rec = sim.fetch()
    v = sim.read_v()
    sim.close()
    return rec.trace, rec.spike_src, rec.spike_step, v


@pytest.mark.parametrize("cells", [9000, 10000, 10400])
def test_tight_packing_changes_nothing(cells):
    low = lowering.lower(workloads.multicomp_net(n_cells=cells, in_degree=20, length_ms=5.0))
    want = _run(low, segments_per_warp=256, kernel_timing=True)
    for a, b in zip(_run(low), want):
        np.testing.assert_array_equal(a, b)
