"""The FP32 net kernels at the edges of their tiles, against FP64.

k_mlp_tiled (energies) and k_mlp_loss_grad (weight gradients) split rows, layer
widths and the sum over inputs into register tiles and staged parts: row counts
around their tiles, widths around 16, 80, 128 and 160 (256 for the gradient) and
odd ones. Tolerances: 1e-5 of the largest energy, 1e-5 (norm) for a gradient,
the FP32 contract of the two entry points.
"""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = {"relu": torch.relu, "tanh": torch.tanh, "silu": torch.nn.functional.silu}


def _layers(dims, seed):
    rng = np.random.default_rng(seed)
    return [(rng.normal(0, 1 / np.sqrt(dims[k]), (dims[k + 1], dims[k])).astype(np.float32),
             rng.normal(0, 0.1, dims[k + 1]).astype(np.float32)) for k in range(len(dims) - 1)]


def _net64(g, layers, act):
    for k, (W, b) in enumerate(layers):
        g = torch.nn.functional.linear(g, W, b)
        if k + 1 < len(layers):
            g = ACTS[act](g)
    return g[:, 0]


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("dims,act", [((47, 150, 150, 1), "relu"), ((121, 160, 144, 1), "tanh"),
                                      ((47, 128, 79, 81, 1), "silu"), ((80, 16, 17, 1), "tanh"), ((160, 1), "relu"),
                                      ((3, 1, 112, 113, 1), "silu")])
def test_tiled_energies(dims, act, rows):
    import gpu_helpers as H
    layers = _layers(dims, 3)
    g = np.random.default_rng(4).normal(0, 1, (rows, dims[0])).astype(np.float32)
    e = H.mlp_energy(layers, act, g)
    ref = _net64(torch.tensor(g).double(), [(torch.tensor(W).double(), torch.tensor(b).double()) for W, b in layers],
                 act).numpy()
    assert np.abs(e - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("rows", [1, 3, 64, 65, 593, 9473])
@pytest.mark.parametrize("dims,act", [((47, 150, 150, 150, 150, 1), "relu"), ((47, 128, 128, 128, 1), "silu"),
                                      ((121, 37, 100, 1), "tanh"), ((47, 256, 200, 1), "silu"), ((5, 1), "tanh"),
                                      ((33, 161, 1), "tanh")])
def test_weight_gradient_tiles(dims, act, rows):
    import gpu_helpers as H
    from amlp._lib import call
    from amlp.engine import EnergyNet
    layers = _layers(dims, 5)
    rng = np.random.default_rng(6)
    g = rng.normal(0, 1, (rows, dims[0])).astype(np.float32)
    y = rng.random(rows).astype(np.float32)
    net = EnergyNet(layers, act, H.DEV)
    gt, yt = H.t32(g), H.t32(y)
    grad = torch.zeros_like(net.d_w)
    loss = torch.zeros(1, dtype=torch.float64, device=H.DEV)
    call("amlp_mlp_loss_grad", gt.data_ptr(), yt.data_ptr(), rows, ctypes.byref(net.struct), grad.data_ptr(),
         loss.data_ptr(), H.stream())
    p = [(torch.tensor(W).double().requires_grad_(), torch.tensor(b).double().requires_grad_()) for W, b in layers]
    l64 = (_net64(torch.tensor(g).double(), p, act) - torch.tensor(y).double()).square().mean()
    ref = torch.cat([t.reshape(-1) for t in torch.autograd.grad(l64, [t for wb in p for t in wb])])
    assert torch.linalg.norm(grad.cpu().double() - ref) <= 1e-5 * torch.linalg.norm(ref)
    assert abs(float(loss.item()) - float(l64)) <= 1e-5 * float(l64)
