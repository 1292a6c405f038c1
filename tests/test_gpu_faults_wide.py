"""Bounded waits of the wide path's net kernels, made to give up on purpose, without any fault.

As ``test_gpu_faults.py`` does for the fused kernel: with the test hook at 0, the first
product wait of every block gives up at once (in the two-tile kernel both teams do, before
their first product). The other roles of that kernel's blocks (weight copies, product
issue) leave with them, what is in flight is drained, the flag is raised and no pair
exerts a force. The next launch at
the normal limit gives the forces of the one before (to the order of the float atomics:
1e-5, norm).
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies", [60, 4000])  # one tile a block, and both teams over two rounds
@pytest.mark.parametrize("shape,phi,widths,act", [
    ("cyl24", 0.35, (128, 128), "silu"),       # two tiles in shared memory
    ("th_v1", 0.005, (160,) * 4, "relu"),      # the first tile in tensor memory, direct-form descriptors
    ("cyl24", 0.35, (150,) * 4, "relu"),
    ("cyl24", 0.35, (96, 96, 96), "tanh"),     # one tile at a time
])
def test_wide_net_wait_that_gives_up(shape, phi, widths, act, bodies):
    import torch
    from amlp import _lib
    from amlp.configs import make_state
    from amlp.engine import EnergyNet, Hypers, System
    _lib.device_error(clear=True)
    net = EnergyNet.xavier(47, widths, act, seed=5)
    s = System(make_state(bodies, shape, phi, seed=3), shape, Hypers(), net, kT=1.0, dt=0.005)
    s.compute_forces("adjoint")
    before = s.F.clone(), s.T.clone()
    assert int(s.nf.item()) > 0 and float(before[0].abs().sum()) > 0.0
    _lib.call("amlp_test_first_wait_limit", 0)
    try:
        s.compute_forces("adjoint")
        torch.cuda.synchronize()
        assert float(s.F.abs().sum()) == 0.0 and float(s.T.abs().sum()) == 0.0
        assert _lib.device_error(clear=False) & 1
    finally:
        _lib.call("amlp_test_first_wait_limit", -1)
        torch.cuda.synchronize()
        _lib.device_error(clear=True)
    s.compute_forces("adjoint")
    torch.cuda.synchronize()
    assert _lib.device_error() == 0
    for got, want in zip((s.F, s.T), before):
        assert float(torch.linalg.norm(got - want)) <= 1e-5 * float(torch.linalg.norm(want))
