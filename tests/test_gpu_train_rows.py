"""A batch that does not fill the training kernel's last tile, for a net that overflows on zero input.

The rows past the last one run on zeros; the batch's own rows keep the first unit
shut (pre-activation -200). Nothing of the former may reach the gradient. Against
FP64 autograd at the entry point's 1e-5 (norm).
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = {"relu": torch.relu, "silu": torch.nn.functional.silu}


@pytest.mark.parametrize("act", ["relu", "silu"])
@pytest.mark.parametrize("rows", [1, 5, 148 * 32 + 1])
def test_rows_past_the_batch_stay_out_of_the_gradient(rows, act):
    import gpu_helpers as H
    from amlp._lib import call
    from amlp.engine import EnergyNet
    rng = np.random.default_rng(8)
    dims = (47, 20, 12, 1)
    layers = [(rng.normal(0, 1 / np.sqrt(dims[k]), (dims[k + 1], dims[k])).astype(np.float32),
               rng.normal(0, 0.1, dims[k + 1]).astype(np.float32)) for k in range(3)]
    g = rng.normal(0, 1, (rows, 47)).astype(np.float32)
    g[:, :2] = 1.0
    layers[0][0][0] = 0.0
    layers[0][0][0, :2] = -2.0 ** 20, -200.0  # exact sums: z = 2^20 - 2^20 - 200 on the batch, 2^20 on zeros
    layers[0][1][0] = 2.0 ** 20
    layers[1][0][0, 0] = 1e33                 # overflows only where the unit is open
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
        if k < 2:
            x = ACTS[act](x)
    l64 = (x[:, 0] - torch.tensor(y).double()).square().mean()
    ref = torch.cat([t.reshape(-1) for t in torch.autograd.grad(l64, [t for wb in p for t in wb])])
    assert torch.isfinite(ref).all()
    assert torch.linalg.norm(grad.cpu().double() - ref) <= 1e-5 * torch.linalg.norm(ref)
    l64 = float(l64.detach())
    assert abs(float(loss.item()) - l64) <= 1e-5 * l64
