"""The gradient kernels at the sizes where they can go wrong: cables of one to a
few compartments, up to and past a block of nodes and a warp's lanes, branching
cells solved by one lane and depth by depth; and a run whose trajectory does not
fit its buffer, which recomputes segments from their checkpoints.

Tolerances: the adjoint against FP64 forward sensitivities contracted with the
same trace gradient, per parameter relative to its largest gradient, 1e-3 (as
tests/test_gpu_gradient.py); recomputed segments repeat the forward's operations
on its checkpoints, so their gradients are equal bit for bit."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.gradient import CableGradient, ParamMap, per_cell_density_map
from eden_gb300.network import ChannelDensity, NetworkSpec, PhysicalCell, Population, PulseInputs, hh_channels
from oracle.cable_grad import Cable

pytestmark = pytest.mark.gpu

GRAD_RTOL = 1e-3


def _cells(parents, length_ms, amp=0.4):
    rng = np.random.default_rng(len(parents[0]))
    spec = NetworkSpec("shapes", 0.025, length_ms, 3, channels=hh_channels())
    for k, parent in enumerate(parents):
        n = len(parent)
        on = np.ones(n, bool)
        dens = [ChannelDensity(0, 0.3, -54.387, on), ChannelDensity(1, 120.0 * rng.uniform(0.9, 1.1), 50.0, on),
                ChannelDensity(2, 36.0, -77.0, on)]
        length, diam = rng.uniform(8.0, 20.0, n), rng.uniform(1.0, 2.0, n)
        length[0] = diam[0] = 20.0
        spec.cells.append(PhysicalCell(f"c{k}", np.asarray(parent), length, diam, dens, cm=1.0, ra=150.0))
        spec.populations.append(Population(f"p{k}", f"c{k}", 1))
    cells = np.arange(len(parents))
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(len(cells)), np.full(len(cells), 100.0),
                                   np.full(len(cells), amp)))
    return lowering.lower(spec)


def _check(low):
    pm = per_cell_density_map(low, [0, 1, 2])
    k = 4
    # the soma and the last compartment of each cell, the soma twice
    rec = np.concatenate([low.phys_comp_off[:-1], low.phys_comp_off[1:] - 1, low.phys_comp_off[:-1]]).astype(np.int32)
    g = CableGradient(low, pm, rec_comp=rec)
    tr = g.forward(pm.values)
    tg = np.cos(np.arange(tr.size, dtype=np.float64)).reshape(tr.shape) + 0.5
    grad = g.backward(tg).reshape(-1, k)
    g.close()
    cab = Cable(low, pm.chan_param, pm.cell_ra_param, low.phys_ra)
    dirs = np.zeros((k, pm.n_params))
    for j in range(k):
        dirs[j, j::k] = 1.0
    tr64, dtr = cab.run(pm.values, low.n_steps, rec, dirs)
    np.testing.assert_allclose(tr, tr64, rtol=0, atol=0.05)
    n = low.n_phys
    ref = np.einsum("nc,jnc->cj", tg.astype(np.float32).astype(np.float64), dtr).reshape(3, n, k).sum(0)
    for j in range(k):
        np.testing.assert_allclose(grad[:, j], ref[:, j], rtol=0, atol=GRAD_RTOL * max(np.abs(ref[:, j]).max(), 1e-12))


@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 9, 32, 33, 64, 65, 130])
def test_cables(n):
    _check(_cells([np.arange(-1, n - 1)] * 2, 4.0))


@pytest.mark.parametrize("n", [3, 40, 200])
def test_trees(n):
    rng = np.random.default_rng(n)
    _check(_cells([workloads.random_tree(rng, n)[0], np.concatenate([[-1], np.zeros(n - 1, np.int64)])], 4.0))


def test_recomputed_segments():
    """30,000 cells over 8,001 steps: 4.8 GB of trajectory, more than is kept."""
    def context(count):
        spec = NetworkSpec("parts", 0.025, 200.0, 3, channels=hh_channels())
        dens = [ChannelDensity(k, c, e, np.ones(1, bool)) for k, c, e in ((0, 0.3, -54.387), (1, 120.0, 50.0), (2, 36.0, -77.0))]
        spec.cells.append(PhysicalCell("c", np.array([-1]), np.array([20.0]), np.array([20.0]), dens, cm=1.0, ra=150.0))
        spec.populations.append(Population("p", "c", count))
        cells = np.arange(count)
        spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(count), np.full(count, 200.0),
                                       0.05 + 0.002 * (cells % 100)))
        low = lowering.lower(spec)
        # one parameter a cell: its sodium conductivity
        chan = np.full(len(low.chan_type), -1, np.int32)
        chan[1::3] = np.arange(count)
        pm = ParamMap(count, chan, np.full(count, -1, np.int32), np.full(count, 120.0, np.float32))
        g = CableGradient(low, pm, rec_comp=np.zeros(1, np.int32))
        tr = g.forward(pm.values)
        grad = g.backward(np.sin(tr))
        g.close()
        return tr, grad
    tr, grad = context(100)
    tr_parts, grad_parts = context(30000)
    assert np.abs(grad[0]) > 0
    np.testing.assert_array_equal(tr_parts, tr)
    np.testing.assert_array_equal(grad_parts[:100], grad)
