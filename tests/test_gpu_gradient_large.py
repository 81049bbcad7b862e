"""Gradients of cells that do not fit shared memory with four steps' coefficients
in flight: two, one, and none (the rows read from global memory, and the forward's
map of the gates too).  A context's launches are shaped by its largest cell, so
small cells beside a large one take its path: their traces and gradients are, bit
for bit, those of a context of their own.  The large cells' own gradients against
FP64 forward sensitivities, as tests/test_gpu_gradient_shapes.py has them (1e-3 of
a parameter's largest)."""
import numpy as np
import pytest

from eden_gb300 import lowering, workloads
from eden_gb300.gradient import CableGradient, per_cell_density_map
from eden_gb300.network import (RATE_EXP, RATE_SIGMOID, Channel, ChannelDensity, Gate, NetworkSpec, PhysicalCell,
                                Population, PulseInputs, Rate, hh_channels)
from oracle.cable_grad import Cable

pytestmark = pytest.mark.gpu

GRAD_RTOL = 1e-3
# compartments, four-gate channels on each beside the HH ones: the floats of two
# steps' coefficients are over 100 kB, of two over what a block may have, of one
LARGE = {"two": (600, 0), "one": (1800, 0), "none": (100, 36)}


def _four_gates():
    gate = lambda name, mid: Gate(name, 1, Rate(RATE_SIGMOID, 0.3, mid, 9.0), Rate(RATE_EXP, 0.2, -60.0, -30.0))
    return Channel("four", [gate(n, -50.0 + 5.0 * k) for k, n in enumerate("abcd")])


def _cell(spec, name, parent, extra):
    rng = np.random.default_rng(len(parent))
    n = len(parent)
    on = np.ones(n, bool)
    dens = [ChannelDensity(0, 0.3, -54.387, on), ChannelDensity(1, 120.0, 50.0, on), ChannelDensity(2, 36.0, -77.0, on)]
    dens += [ChannelDensity(3, 0.01 * (1 + k % 3), -70.0, on) for k in range(extra)]
    length, diam = rng.uniform(8.0, 20.0, n), rng.uniform(1.0, 2.0, n)
    length[0] = diam[0] = 20.0
    spec.cells.append(PhysicalCell(name, np.asarray(parent), length, diam, dens, cm=1.0, ra=150.0))
    spec.populations.append(Population("p" + name, name, 1))


def _network(large=None, small=True, length_ms=3.0):
    spec = NetworkSpec("large", 0.025, length_ms, 3, channels=hh_channels() + [_four_gates()])
    if small:
        _cell(spec, "chain", np.arange(-1, 39), 0)
        _cell(spec, "tree", workloads.random_tree(np.random.default_rng(5), 70)[0], 0)
        _cell(spec, "active", workloads.random_tree(np.random.default_rng(6), 20)[0], 2)
    if large:
        _cell(spec, "large", workloads.random_tree(np.random.default_rng(7), large[0])[0], large[1])
    n = len(spec.cells)
    cells = np.arange(n)
    spec.pulses.append(PulseInputs("*", cells, 0 * cells, np.zeros(n), np.full(n, 100.0), np.full(n, 0.4)))
    return lowering.lower(spec)


def _gradient(low):
    pm = per_cell_density_map(low, [0, 1, 2])
    # the soma twice, and the last compartment, of each cell
    rec = np.stack([low.phys_comp_off[:-1], low.phys_comp_off[1:] - 1, low.phys_comp_off[:-1]], 1).ravel().astype(np.int32)
    g = CableGradient(low, pm, rec_comp=rec)
    try:
        tr = g.forward(pm.values)
        steps, cols = np.arange(len(tr))[:, None], np.arange(len(rec))[None, :]
        tg = np.cos(0.7 * steps + cols) + 0.5
        return pm, rec, tr, tg, g.backward(tg)
    finally:
        g.close()


@pytest.mark.parametrize("large", list(LARGE))
def test_beside_a_large_cell(large):
    _, rec, tr, _, grad = _gradient(_network())
    _, _, tr1, _, grad1 = _gradient(_network(LARGE[large]))
    assert np.abs(grad).min() > 0
    np.testing.assert_array_equal(tr1[:, :len(rec)], tr)
    np.testing.assert_array_equal(grad1[:len(grad)], grad)


@pytest.mark.parametrize("large", list(LARGE))
def test_a_large_cell(large):
    low = _network(LARGE[large], small=False, length_ms=1.5)
    pm, rec, tr, tg, grad = _gradient(low)
    cab = Cable(low, pm.chan_param, pm.cell_ra_param, low.phys_ra)
    tr64, dtr = cab.run(pm.values, low.n_steps, rec, np.eye(pm.n_params))
    np.testing.assert_allclose(tr, tr64, rtol=0, atol=0.05)
    ref = np.einsum("nc,jnc->j", tg.astype(np.float32).astype(np.float64), dtr)
    np.testing.assert_allclose(grad, ref, rtol=GRAD_RTOL, atol=0)
