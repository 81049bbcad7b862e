"""Contexts alive at the same time share their kernels: one created later with
smaller cells must not keep an earlier one, which needs more shared memory,
from launching."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import MODE_BATCHED, MODE_PLAIN, Simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [MODE_PLAIN, MODE_BATCHED], ids=["plain", "batched"])
def test_smaller_context_created_later(mode):
    large, small = (lowering.lower(workloads.multicomp_net(n_cells=12, in_degree=5, length_ms=10.0, max_seg=m))
                    for m in (500, 8))
    alone = Simulation(large, mode=mode)
    want = alone.run()
    alone.close()
    first, second = Simulation(large, mode=mode), Simulation(small, mode=mode)
    second.run()
    got = first.run()
    first.close()
    second.close()
    np.testing.assert_array_equal(got.trace, want.trace)
    np.testing.assert_array_equal(got.spike_step, want.spike_step)
