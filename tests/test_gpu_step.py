"""The step's combined launches against the single ones, to the bit.

``amlp_nvt_step`` against ``amlp_nvt_step_two`` then ``amlp_nvt_step_one`` over
three steps at sizes around the block of 256 (the kinetic energies of the
many-system form are sums of FP64 atomics: relative 1e-12), and
``amlp_pair_filter_zero`` against ``amlp_pair_filter`` with the sums it zeroes.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(n, seed):
    import torch
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g)
    q = r(n, 4)
    t = {"pos": 9.0 * (torch.rand(n, 3, generator=g) - 0.5), "vel": r(n, 3), "accel": torch.zeros(n, 3),
         "quat": q / q.norm(dim=1, keepdim=True), "angmom": r(n, 4), "dp": torch.zeros(n, 4),
         "mass": 0.5 + torch.rand(n, generator=g), "F": 5.0 * r(n, 3), "T": 5.0 * r(n, 3)}
    return {k: v.float().contiguous().cuda() for k, v in t.items()}


def _prm(n, nve):
    from amlp._lib import Nvt
    prm = Nvt()
    prm.dt, prm.tau, prm.kT, prm.n_dof, prm.rn_dof = 0.005, 0.5, 1.1, 3.0 * (n - 1) or 3.0, 3.0 * n
    prm.moi[0], prm.moi[1], prm.moi[2] = 0.2, 0.3, 0.4
    prm.box, prm.nve = 9.0, nve
    return prm


def _th(count):
    import torch
    from amlp._lib import Thermostat
    th = Thermostat()
    th.xi, th.eta, th.xi_rot, th.eta_rot, th.thermo_fac = (-0.0317711, 0.108609, 0.00814227, -0.014238, 1.00011)
    th.ke_t, th.ke_r, th.pe = 3.0, 2.0, 7.0
    return torch.frombuffer(bytearray(bytes(th) * count), dtype=torch.uint8).cuda()


def _p(t, *names):
    return [t[k].data_ptr() for k in names]


@pytest.mark.parametrize("nve", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_step_equals_step_two_then_step_one(n, nve):
    import torch
    import gpu_helpers as gh
    from amlp._lib import call, size_query
    a, b, prm, ta, tb = _state(n, 3), _state(n, 3), _prm(n, nve), _th(1), _th(1)
    ws = [torch.zeros(size_query("amlp_nvt_workspace_bytes", n), dtype=torch.uint8, device="cuda") for _ in range(2)]
    tail = [n, ctypes.byref(prm)]
    for _ in range(3):
        call("amlp_nvt_step_two", *_p(a, "vel", "accel", "F", "mass", "quat", "T", "angmom", "dp"), *tail,
             ta.data_ptr(), gh.stream())
        call("amlp_nvt_step_one", *_p(a, "pos", "vel", "accel", "quat", "angmom", "dp", "mass"), *tail, ta.data_ptr(),
             ws[0].data_ptr(), ws[0].numel(), gh.stream())
        call("amlp_nvt_step", *_p(b, "pos", "vel", "accel", "quat", "angmom", "dp", "mass", "F", "T"), *tail,
             tb.data_ptr(), ws[1].data_ptr(), ws[1].numel(), gh.stream())
    for k in a:
        assert torch.equal(a[k], b[k]), k
    assert torch.equal(ta, tb)
    assert int(ws[1][:4].sum()) == 0


@pytest.mark.parametrize("sizes", [(1, 1), (31, 257, 5), (256, 300)])
def test_multi_step_equals_step_two_then_step_one(sizes):
    import torch
    import gpu_helpers as gh
    from amlp._lib import Replica, Thermostat, call
    n, nrep = sum(sizes) + 3, len(sizes) + 1  # three free bodies, one free system
    a, b, prm, ta, tb = _state(n, 4), _state(n, 4), _prm(n, 0), _th(nrep), _th(nrep)
    rep = np.full(n, -1, np.int32)
    rep[:sum(sizes)] = np.repeat(np.arange(len(sizes), dtype=np.int32), sizes)
    rep = torch.tensor(rep, device="cuda")
    reps = (Replica * nrep)()
    for k, m in enumerate(sizes):
        reps[k].kT, reps[k].n_dof, reps[k].rn_dof, reps[k].box, reps[k].nve = 1.0 + k, 3.0 * m, 3.0 * m, 9.0 - k, k & 1
    rp = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).cuda()
    end = [rp.data_ptr(), ctypes.byref(prm)]
    call("amlp_multi_nvt_step_two", *_p(a, "vel", "accel", "F", "mass", "quat", "T", "angmom", "dp"), rep.data_ptr(),
         n, nrep, *end, ta.data_ptr(), gh.stream())
    call("amlp_multi_nvt_step_one", *_p(a, "pos", "vel", "accel", "quat", "angmom", "dp", "mass"), rep.data_ptr(), n,
         *end, ta.data_ptr(), gh.stream())
    call("amlp_multi_nvt_step", *_p(b, "pos", "vel", "accel", "quat", "angmom", "dp", "mass", "F", "T"),
         rep.data_ptr(), n, nrep, *end, tb.data_ptr(), gh.stream())
    for k in a:
        assert torch.equal(a[k], b[k]), k
    for x, y in zip((Thermostat * nrep).from_buffer_copy(bytes(ta.cpu().numpy().tobytes())),
                    (Thermostat * nrep).from_buffer_copy(bytes(tb.cpu().numpy().tobytes()))):
        for f in ("xi", "eta", "xi_rot", "eta_rot", "thermo_fac", "pe"):
            assert getattr(x, f) == getattr(y, f), f
        for f in ("ke_t", "ke_r"):
            assert abs(getattr(x, f) - getattr(y, f)) <= 1e-12 * abs(getattr(x, f)), f


@pytest.mark.parametrize("n", [1, 700, 60000])
def test_pair_filter_zero(n):
    import torch
    import gpu_helpers as gh
    from amlp._lib import call, size_query
    g = torch.Generator().manual_seed(n)
    pos = (9.0 * (torch.rand(n, 3, generator=g) - 0.5)).cuda()
    cap = 5 * n
    vp = torch.randint(0, n, (cap, 2), generator=g, dtype=torch.int32).cuda()
    nv = torch.tensor([cap - 1], dtype=torch.int64, device="cuda")
    ws = torch.empty(size_query("amlp_filter_workspace_bytes", cap), dtype=torch.uint8, device="cuda")
    out = [torch.zeros(cap, 2, dtype=torch.int32, device="cuda") for _ in range(2)]
    cnt = [torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(2)]
    F, T = torch.full((n + 1, 3), 3.0, device="cuda"), torch.full((n + 1, 3), 3.0, device="cuda")
    pe = torch.full((2,), 3.0, dtype=torch.float64, device="cuda")
    head = [pos.data_ptr(), 9.0, 2.5, vp.data_ptr(), nv.data_ptr(), cap]
    call("amlp_pair_filter", *head, out[0].data_ptr(), cnt[0].data_ptr(), ws.data_ptr(), ws.numel(), gh.stream())
    call("amlp_pair_filter_zero", *head, out[1].data_ptr(), cnt[1].data_ptr(), ws.data_ptr(), ws.numel(),
         F.data_ptr(), T.data_ptr(), n, pe.data_ptr(), gh.stream())
    assert torch.equal(out[0], out[1]) and torch.equal(cnt[0], cnt[1])
    for t in (F, T):
        assert float(t[:n].abs().max()) == 0.0 and bool((t[n] == 3.0).all())
    assert float(pe[0]) == 0.0 and float(pe[1]) == 3.0
