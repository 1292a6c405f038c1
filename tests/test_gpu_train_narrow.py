"""The training kernel's narrow form (nets at most 16 wide, inputs included) and the line to the wide one.

Widths on both sides of 16, row counts at the edges of a tile and of the four blocks per SM,
against FP64 autograd at the entry point's 1e-5 (norm).
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = {"relu": torch.relu, "tanh": torch.tanh, "silu": torch.nn.functional.silu}


@pytest.mark.parametrize("rows", [1, 3, 64, 65, 4 * 148 * 64 + 1])
@pytest.mark.parametrize("dims,act", [((1, 3, 1), "relu"), ((16, 1), "tanh"), ((16, 16, 16, 1), "silu"),
                                      ((16, 17, 1), "silu"), ((17, 16, 1), "relu"), ((5, 9, 16, 2, 13, 1), "tanh"),
                                      ((16,) * 8 + (1,), "silu")])
def test_narrow_weight_gradients(dims, act, rows):
    import gpu_helpers as H
    from amlp._lib import call
    from amlp.engine import EnergyNet
    rng = np.random.default_rng(12)
    layers = [(rng.normal(0, 1 / np.sqrt(dims[k]), (dims[k + 1], dims[k])).astype(np.float32),
               rng.normal(0, 0.1, dims[k + 1]).astype(np.float32)) for k in range(len(dims) - 1)]
    g = rng.normal(0, 1, (rows, dims[0])).astype(np.float32)
    y = rng.random(rows).astype(np.float32)
    net = EnergyNet(layers, act, H.DEV)
    gt, yt = H.t32(g), H.t32(y)
    grad = torch.zeros_like(net.d_w)
    loss = torch.zeros(1, dtype=torch.float64, device=H.DEV)
    call("amlp_mlp_loss_grad", gt.data_ptr(), yt.data_ptr(), rows, ctypes.byref(net.struct), grad.data_ptr(),
         loss.data_ptr(), H.stream())
    p = [(torch.tensor(W).double().requires_grad_(), torch.tensor(b).double().requires_grad_()) for W, b in layers]
    x = torch.tensor(g).double()
    for k, (W, b) in enumerate(p):
        x = torch.nn.functional.linear(x, W, b)
        if k + 1 < len(p):
            x = ACTS[act](x)
    l64 = (x[:, 0] - torch.tensor(y).double()).square().mean()
    ref = torch.cat([t.reshape(-1) for t in torch.autograd.grad(l64, [t for wb in p for t in wb])])
    l64 = float(l64.detach())
    assert torch.linalg.norm(grad.cpu().double() - ref) <= 1e-5 * torch.linalg.norm(ref)
    assert abs(float(loss.item()) - l64) <= 1e-5 * l64
