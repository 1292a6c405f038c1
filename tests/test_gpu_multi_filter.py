"""The many-system pair filters against the single-system one, to the bit.

Systems with boxes of their own, free body slots between them and a free system:
``amlp_multi_pair_filter`` and ``amlp_multi_pair_filter_zero`` give each system the
pairs of ``amlp_pair_filter`` on it alone, and the second zeroes exactly the sums
it is told to.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(2,), (5, 700, 31), (20000, 300, 9000)])
def test_multi_pair_filters(sizes):
    import torch
    import gpu_helpers as H
    from amlp._lib import Replica, call, size_query
    rng = np.random.default_rng(sum(sizes))
    nrep, free, cutoff = len(sizes) + 1, 3, 2.5  # the last system is free, `free` body slots follow each
    reps = (Replica * nrep)()
    pos, rep, vp, expect, start = [], [], [], [], 0
    for k, m in enumerate(sizes):
        L = float(np.float32(7.0 + k))
        reps[k].box, reps[k].n_dof = L, 3.0 * m
        x = rng.uniform(-L / 2, L / 2, (m, 3)).astype(np.float32)
        v = rng.integers(0, m, (4 * m + 1, 2))
        expect.append(H.pair_filter(x, L, cutoff, v) + start)
        pos += [x, np.zeros((free, 3), np.float32)]
        rep += [np.full(m, k), np.full(free, -1)]
        vp.append(v + start)
        start += m + free
    n = start
    pos, rep = H.t32(np.concatenate(pos)), torch.tensor(np.concatenate(rep).astype(np.int32), device=H.DEV)
    vp = torch.tensor(np.concatenate(vp).astype(np.int32), device=H.DEV).contiguous()
    expect = np.concatenate(expect)
    rp = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).to(H.DEV)
    cap = vp.shape[0]
    nv = torch.tensor([cap], dtype=torch.int64, device=H.DEV)
    ws = torch.empty(size_query("amlp_filter_workspace_bytes", cap), dtype=torch.uint8, device=H.DEV)
    F, T = torch.full((n + 1, 3), 3.0, device=H.DEV), torch.full((n + 1, 3), 3.0, device=H.DEV)
    pe = torch.full((nrep + 1,), 3.0, dtype=torch.float64, device=H.DEV)
    for name, tail in (("amlp_multi_pair_filter", []),
                       ("amlp_multi_pair_filter_zero", [F.data_ptr(), T.data_ptr(), n, pe.data_ptr(), nrep])):
        out = torch.full((cap, 2), -1, dtype=torch.int32, device=H.DEV)
        cnt = torch.zeros(1, dtype=torch.int64, device=H.DEV)
        call(name, pos.data_ptr(), rep.data_ptr(), rp.data_ptr(), cutoff, vp.data_ptr(), nv.data_ptr(), cap,
             out.data_ptr(), cnt.data_ptr(), ws.data_ptr(), ws.numel(), *tail, H.stream())
        assert int(cnt.item()) == len(expect)
        assert np.array_equal(out[:len(expect)].cpu().numpy(), expect)
        assert float(F[:n].abs().max()) == (0.0 if tail else 3.0)
    for t in (F, T):
        assert float(t[:n].abs().max()) == 0.0 and bool((t[n] == 3.0).all())
    assert float(pe[:nrep].abs().max()) == 0.0 and float(pe[nrep]) == 3.0
