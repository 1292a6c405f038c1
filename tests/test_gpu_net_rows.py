"""Single rows of the wide force path's net pass at the edges of its tiles and rounds.

Sums over all pairs hardly move when one row is lost. Here each row at an edge (the
first and last of the first and last tile, of tiles 147, 148, 295 and 296) is a pair of
two bodies that no other pair uses, in a system of its own, so its force, torques and
energy stand alone. They are the list's strongest pairs below the clip of 100. Against FP64 autograd:
forces and torques within 2e-3 of the largest component (at least 1), as for the single
pair of ``test_gpu_tiles.py``; energies within 1e-3 (at least 1e-3), far below the energy itself.
"""
import ctypes

import numpy as np
import pytest

from test_gpu_net_pairs import HYPERS, SHAPE, _pairs

pytestmark = pytest.mark.gpu


def _edge_rows(count):
    rows = {r for t in (0, 147, 148, 295, 296, (count - 1) // 128) for r in (128 * t, 128 * t + 127)}
    return sorted({r for r in rows if r < count} | {count - 1})


@pytest.mark.parametrize("count", [1, 128, 129, 148 * 128 - 1, 148 * 128 + 1, 296 * 128, 296 * 128 + 1])
@pytest.mark.parametrize("widths,act", [
    ((128, 128), "silu"),             # two tiles in shared memory, act' in tensor memory
    ((64, 80, 48, 64), "relu"),       # two tiles in shared memory
    ((150,), "relu"),                 # one layer: its weights stay
    ((160, 160, 160, 160), "relu"),   # the first tile in tensor memory
    ((96, 96, 96), "tanh"),           # one tile at a time
])
def test_rows_at_round_edges(widths, act, count):
    import gpu_helpers as H
    import torch
    from amlp._lib import Replica, call, size_query
    from amlp.engine import EnergyNet
    from oracle import adjoint
    from oracle.shapes import SHAPES
    layers = EnergyNet.xavier(47, widths, act, seed=5, device="cpu").layers
    s, base = _pairs(layers, act)
    ex = adjoint.exact_pair_forces(s.pos, s.orient, base, s.L, SHAPES[SHAPE], HYPERS, layers, act)
    rows = _edge_rows(count)
    size = np.abs(np.concatenate([ex[q] for q in ("F_pair", "T_i", "T_j")], 1)).max(1)
    strong = np.argsort(np.where(size < 95.0, -np.abs(ex["F_pair"]).max(1), 0.0))[:len(rows)]
    assert np.abs(ex["F_pair"][strong]).max(1).min() > 1.0 and np.abs(ex["E"][strong]).min() > 0.1
    n, k = len(s.pos), len(rows)
    pairs = np.concatenate([base] * (count // len(base) + 1))[:count]
    pairs[rows] = n + np.arange(2 * k).reshape(k, 2)
    body = np.concatenate([np.arange(n), base[strong].reshape(-1)])
    rep = np.concatenate([np.zeros(n, np.int32), 1 + np.repeat(np.arange(k, dtype=np.int32), 2)])
    reps = (Replica * (k + 1))()
    for r in reps:
        r.box = float(s.L)
    dev = dict(device=H.DEV)
    pos, quat, pts = H.t32(s.pos[body]), H.t32(s.orient[body]), H.t32(SHAPES[SHAPE]["pts"])
    rep, pr = torch.tensor(rep, **dev), torch.tensor(pairs.astype(np.int32), **dev).contiguous()
    rp = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).to(H.DEV)
    cnt = torch.tensor([count], dtype=torch.int64, **dev)
    F, T = torch.zeros(n + 2 * k, 3, **dev), torch.zeros(n + 2 * k, 3, **dev)
    pe = torch.zeros(k + 1, dtype=torch.float64, **dev)
    ws = torch.empty(size_query("amlp_adjoint_workspace_bytes", count), dtype=torch.uint8, **dev)
    nep, net = H.nep_struct(SHAPES[SHAPE], HYPERS, pts), EnergyNet(layers, act, H.DEV)
    call("amlp_multi_forces_adjoint_wide", pos.data_ptr(), quat.data_ptr(), rep.data_ptr(), rp.data_ptr(),
         pr.data_ptr(), cnt.data_ptr(), count, ctypes.byref(nep), ctypes.byref(net.struct), F.data_ptr(), T.data_ptr(),
         pe.data_ptr(), ws.data_ptr(), ws.numel(), H.stream())
    F, T, pe = F.cpu().numpy(), T.cpu().numpy(), pe.cpu().numpy()
    for e, b in enumerate(strong):
        i, j = n + 2 * e, n + 2 * e + 1
        for got, ref in ((F[i], ex["F_pair"][b]), (F[j], -ex["F_pair"][b]), (T[i], ex["T_i"][b]), (T[j], ex["T_j"][b])):
            np.testing.assert_allclose(got, ref, rtol=0, atol=2e-3 * max(1.0, np.abs(ref).max()), err_msg=str(rows[e]))
        assert abs(pe[1 + e] - ex["E"][b]) <= 1e-3 * max(1.0, abs(ex["E"][b])), rows[e]
