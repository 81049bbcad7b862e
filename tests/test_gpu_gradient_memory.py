"""The gradient contexts' device memory: buffers cut to what a caller allows or to
what the device has left, and the same results with them.

A trace does not depend on them: equal bit for bit.  Of a gradient only the order
of its double-precision sums does: a float's last place (2^-23 of a value, twice
for two roundings), and 1e-9 of the largest gradient where terms cancel (sums of
some 10,000 doubles: 10,000 * 2^-53 of their absolute values, 1e-12, times a
thousand)."""
import numpy as np
import pytest
import torch

from eden_gb300 import lowering, workloads
from eden_gb300.gradient import CableGradient, per_cell_density_map, with_weights

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _gradient(low, pm, rec, **options):
    g = CableGradient(low, pm, rec_comp=rec, **options)
    try:
        tr = g.forward(pm.values)
        tg = np.cos(np.arange(tr.size, dtype=np.float64)).reshape(tr.shape) + 0.25
        return tr, g.backward(tg)
    finally:
        g.close()


def _row_bytes(low):
    gates = sum(int(low.chan_types[t]["n_gates"]) for t in low.chan_type)
    return 4 * (2 * low.n_comp + gates)


@pytest.mark.parametrize("checkpoint_every", [37, 100])
@pytest.mark.parametrize("drive", [0, 6])
def test_in_parts_as_in_whole(drive, checkpoint_every):
    low = lowering.lower(workloads.ball_and_stick(n_inst=9, n_dend=30, length_ms=30.0, syn_drive=drive))
    pm = per_cell_density_map(low, [0, 1, 2])
    if drive:
        pm = with_weights(low, pm)
    rec = np.concatenate([low.phys_comp_off[:-1], low.phys_comp_off[1:] - 1]).astype(np.int32)
    # more than one group of segments, block of coefficients and block of exposures
    assert low.n_steps * _row_bytes(low) > 2 * (MIB // 2)
    items = len(low.syn_target) + len(low.timed_target)
    assert not drive or low.n_steps * 4 * items > MIB // 16
    tr, grad = _gradient(low, pm, rec, checkpoint_every=checkpoint_every)
    tr1, grad1 = _gradient(low, pm, rec, checkpoint_every=checkpoint_every, buffer_mib=1)
    np.testing.assert_array_equal(tr1, tr)
    assert np.abs(grad).max() > 0
    np.testing.assert_allclose(grad1, grad, rtol=2.0 ** -22, atol=1e-9 * np.abs(grad).max())


def _long_run():
    """64 cables over 8,001 steps: 0.6 GB of trajectory, 1.3 GB of coefficients."""
    low = lowering.lower(workloads.ball_and_stick(n_inst=64, n_dend=50, length_ms=200.0))
    pm = per_cell_density_map(low, [0, 1, 2])
    return low, pm, low.phys_comp_off[:-1].astype(np.int32)


def test_takes_what_it_is_allowed():
    low, pm, rec = _long_run()
    torch.cuda.synchronize()
    _gradient(low, pm, rec, buffer_mib=16)   # what the library itself takes on first use
    before = torch.cuda.mem_get_info(0)[0]
    g = CableGradient(low, pm, rec_comp=rec, buffer_mib=16)
    used = before - torch.cuda.mem_get_info(0)[0]
    g.close()
    # 80 checkpoints, trace and its gradient, and 2 MiB of granularity for each array
    fixed = 81 * _row_bytes(low) + 2 * 4 * low.n_steps * len(rec)
    assert used < 16 * MIB + fixed + 64 * 2 * MIB


def test_beside_a_program_that_holds_the_device():
    low, pm, rec = _long_run()
    want = _gradient(low, pm, rec)
    torch.cuda.empty_cache()
    hold = [torch.empty(torch.cuda.mem_get_info(0)[0] - 1024 * MIB, dtype=torch.uint8, device="cuda")]
    try:
        got = _gradient(low, pm, rec)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_allclose(got[1], want[1], rtol=2.0 ** -22, atol=1e-9 * np.abs(want[1]).max())
