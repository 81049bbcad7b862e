"""A window's kernels that start while the one before drains compute the same
bits as ones that do not: timing each kernel puts events between them, which
order them completely.  Windows of one step and of many, in both modes, a small
network and one whose input kernel fills the GPU, and many runs in a row."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.engine import MODE_BATCHED, MODE_PLAIN, Simulation

pytestmark = pytest.mark.gpu

NETWORKS = {"trees": lambda: workloads.multicomp_net(n_cells=60, in_degree=20, length_ms=10.0, max_seg=80, n_recorded=6,
                                                     hh_dend_frac=0.2, syn_on_dendrites=True),
            "mixed": lambda: workloads.mixed_scale(n_izh=12000, n_mc=600, in_degree=20, length_ms=10.0, n_seg=30)}


def _run(low, pieces, **options):
    sim = Simulation(low, **options)
    sim.initialize()
    out = []
    for n in pieces:
        sim.run_steps(n)
        rec = sim.fetch()
        out += [rec.trace, rec.spike_src, rec.spike_step, sim.read_v()]
    sim.close()
    return out


@pytest.mark.parametrize("options", [dict(), dict(steps_per_launch=1), dict(mode=MODE_PLAIN), dict(codegen=-1)], ids=str)
@pytest.mark.parametrize("network", list(NETWORKS))
def test_early_start_changes_nothing(network, options):
    low = lowering.lower(NETWORKS[network]())
    pieces = [200, 40, 20, 120]
    want = _run(low, pieces, kernel_timing=True, **options)
    got = _run(low, pieces, **options)
    assert sum(len(a) for a in want[1::4]) > 0
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
