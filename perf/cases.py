"""The work whose speed counts, as cases through the public entry points.

The framework's users run rigid-body NVT simulations with a pair-energy net (one
system, or many small ones in a pool), differentiate pair energies and train the
net. The cases are the parts those programs spend their time in, each through
the call such a program makes:

* ``forces``  ``System.compute_forces``: pair filter and force pass of one step
              ("adjoint" is the analytic method, "fd" and "fd_split" the
              reference's finite differences, the drop-in modules' default);
* ``run``     ``System.run``: 10 NVT steps from a given state, a Verlet rebuild every 100 steps;
* ``pool``    ``NativePool``: requests admitted, advanced by one segment, evicted;
* ``nlist``   ``amlp_nlist_build``: the Verlet list into the caller's buffer;
* ``vjp``     ``amlp.autograd.pair_energies`` forward and backward to positions,
              orientations and weights;
* ``train``   ``amlp.autograd.mse_loss_grad``: loss and weight gradient of a batch.

Bodies start on the jittered lattice of ``amlp.configs`` at the packing fractions
(or the number density) of the benchmark's workloads, with that workload's net.
Inputs depend on the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "anisotropic-ml_b200"))

from amlp.autograd import PairModel, mse_loss_grad, pair_energies  # noqa: E402
from amlp.configs import make_state  # noqa: E402
from amlp.engine import EnergyNet, Hypers, System  # noqa: E402
from amlp.native import NativePool  # noqa: E402
from amlp._lib import Thermostat, call, size_query  # noqa: E402
from amlp.shapes import get_shape  # noqa: E402

# The benchmark's workloads: shape, packing fraction (or bodies per volume), hypers, net
# ("xavier": seeded weights; a name: the weights stored under tests/golden) and activation.
SYSTEMS = {
    "cube26": dict(shape="cube26", phi=0.45, hypers=(10, 8, 4), net="xavier", widths=(64, 64), act="tanh"),
    "cyl24": dict(shape="cyl24", phi=0.35, hypers=(10, 8, 4), net="model_cyl24_soft", widths=(128, 128), act="silu"),
    "tetra16": dict(shape="tetra16", phi=0.40, hypers=(10, 8, 4), net="model_tetra16_soft", widths=(128,) * 3,
                    act="silu"),
    "th_C104": dict(shape="th_v1", rho=200 / 33.0 ** 3, hypers=(10, 8, 4), net="model_th_C104", widths=(150,) * 4,
                    act="relu"),
    "th_C100": dict(shape="th_v1", rho=200 / 33.0 ** 3, hypers=(10, 10, 10), net="model_th_C100", widths=(150,) * 4,
                    act="relu"),
}
SKIN = 2.0        # System's default: the Verlet radius is the pair cutoff plus this
RUN_STEPS = 10    # steps per System.run and per pool segment: short, since trajectories of
POOL_STEPS = 10   # hard bodies part exponentially (rounding grows e^10 in 100 steps of a stiff net)


def listed():
    return [
        # the benchmark's step: 131,072 cubes, the force pass that is 95 % of it
        dict(name="forces_cube26_131072", kind="forces", system="cube26", method="adjoint", n=131072),
        # a small system stepped by a host program: one force pass is a few tiles, launches count
        dict(name="forces_cube26_1000", kind="forces", system="cube26", method="adjoint", n=1000),
        # cylinders with the trained 128-wide SiLU net, beyond the fused kernel's width (odd size)
        dict(name="forces_cyl24_60001", kind="forces", system="cyl24", method="adjoint", n=60001),
        # the reference's own trained 150 x 4 ReLU models on tetrahedra, analytic forces, D = 47 and 121
        dict(name="forces_th_C104_262144", kind="forces", system="th_C104", method="adjoint", n=262144),
        dict(name="forces_th_C100_99991", kind="forces", system="th_C100", method="adjoint", n=99991),
        # the drop-in's default forces: fused finite differences (nets up to 64 wide) ...
        dict(name="fd_cube26_20011", kind="forces", system="cube26", method="fd", n=20011),
        # ... and the reference's data flow for the shipped 150-wide models
        dict(name="fd_split_th_C104_65536", kind="forces", system="th_C104", method="fd_split", n=65536),
        # a whole simulation call on the 1,000-cube configuration: graph replay, both NVT halves
        dict(name="run_cube26_1000", kind="run", system="cube26", n=1000),
        # serving: six requests of mixed sizes through one segment
        dict(name="pool_cube26_6x3000", kind="pool", system="cube26", n=3000, count=6),
        # the Verlet rebuild of the benchmark's system (11 million pairs)
        dict(name="nlist_cube26_131072", kind="nlist", system="cube26", n=131072),
        # differentiable pair energies: 50,021 pairs of 16-point tetrahedra, forward and backward
        dict(name="vjp_tetra16_50021", kind="vjp", system="tetra16", pairs=50021),
        # a training batch of the reference's 150 x 4 ReLU net
        dict(name="train_th_C104_16384", kind="train", system="th_C104", rows=16384),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# Largest drawn size of each kind and system, so that no drawn case costs more than the largest listed one.
_MOST_BODIES = {("adjoint", "cube26"): 131072, ("adjoint", "cyl24"): 100000, ("adjoint", "tetra16"): 12000,
                ("adjoint", "th_C104"): 262144, ("adjoint", "th_C100"): 262144, ("fd", "cube26"): 24000,
                ("fd_split", "th_C104"): 40000, ("fd_split", "th_C100"): 40000}


def draw(rng):
    kind = rng.choice(["forces", "forces", "forces", "forces", "run", "pool", "nlist", "vjp", "train"])
    if kind == "forces":
        method, system = rng.choice(sorted(_MOST_BODIES))
        least = 200 if system.startswith("th") else 500
        return dict(kind=kind, system=system, method=method, n=_log_uniform(rng, least, _MOST_BODIES[method, system]))
    if kind == "run":
        return dict(kind=kind, system="cube26", n=_log_uniform(rng, 500, 5000))
    if kind == "pool":
        return dict(kind=kind, system="cube26", n=_log_uniform(rng, 500, 5000), count=rng.randint(1, 6))
    if kind == "nlist":
        system = rng.choice(["cube26", "cyl24", "tetra16", "th_C104"])
        return dict(kind=kind, system=system, n=_log_uniform(rng, 500, 20000 if system == "tetra16" else 131072))
    if kind == "vjp":
        return dict(kind=kind, system=rng.choice(["cube26", "cyl24", "tetra16"]), pairs=_log_uniform(rng, 500, 100000))
    return dict(kind=kind, system=rng.choice(["cube26", "cyl24", "tetra16", "th_C104", "th_C100"]),
                rows=_log_uniform(rng, 64, 32768))


# ------------------------------------------------------------------ inputs
def _layers(case, seed):
    """The net as (W, b) arrays. ``run`` and ``pool`` take the Xavier net with its output
    layer scaled by 0.01: a random net's full-size forces are not a physical potential."""
    sysd = SYSTEMS[case["system"]]
    if sysd["net"] != "xavier":
        z = np.load(os.path.join(_ROOT, "tests", "golden", sysd["net"] + ".npz"))
        return [(z["W%d" % k], z["b%d" % k]) for k in range(len(z.files) // 2)]
    layers = EnergyNet.xavier(Hypers(*sysd["hypers"]).D, sysd["widths"], sysd["act"], seed, "cpu").layers
    if case["kind"] in ("run", "pool"):
        W, b = layers[-1]
        layers[-1] = (W * np.float32(0.01), b)
    return layers


def _state(case, n, seed):
    sysd = SYSTEMS[case["system"]]
    if "rho" in sysd:
        return make_state(n, sysd["shape"], 0.0, kT=0.5, seed=seed, L=(n / sysd["rho"]) ** (1 / 3))
    return make_state(n, sysd["shape"], sysd["phi"], kT=1.0, seed=seed)


def _system(case, seed):
    sysd = SYSTEMS[case["system"]]
    net = EnergyNet(_layers(case, seed), sysd["act"], "cuda")
    return System(_state(case, case["n"], seed), sysd["shape"], Hypers(*sysd["hypers"]), net,
                  kT=0.5 if "rho" in sysd else 1.0, dt=0.005)


def _pairs_within(pos, L, cutoff):
    """Pairs (i, j), i < j, whose FP32 minimum-image distance is below the cutoff, sorted
    by (i, j): the reference's filter (DescriptorGenerator.py:168-182) on all pairs."""
    L32 = torch.tensor(np.float32(L), device=pos.device)
    half = L32 * 0.5
    n, out = pos.shape[0], []
    rows = max(1, (1 << 26) // n)
    for a in range(0, n, rows):
        m = min(n, a + rows) - a
        d2 = torch.zeros(m, n - a, device=pos.device)
        for k in range(3):
            d = pos[None, a:, k] - pos[a:a + m, None, k]
            d = torch.where(d > half, d - L32, d)
            d = torch.where(d < -half, L32 + d, d)
            d2 += d * d
        keep = torch.nonzero((d2.sqrt().double() < cutoff).triu(1))
        out.append(keep + a)
    return torch.cat(out)


def _pair_inputs(case, count, seed):
    """A minibatch of ``count`` pairs drawn from a small system, in (i, j) order."""
    sysd = SYSTEMS[case["system"]]
    shape = get_shape(sysd["shape"])
    rho = sysd.get("rho") or sysd["phi"] / shape.volume
    per_body = 2 / 3 * math.pi * rho * shape.cutoff ** 3
    n = max(int(1.5 * count / per_body) + 1, int(rho * (2.2 * shape.cutoff) ** 3) + 1)
    state = _state(case, n, seed)
    pos = torch.tensor(state.pos, device="cuda")
    quat = torch.tensor(state.orient, device="cuda")
    pairs = _pairs_within(pos, state.L, shape.cutoff)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pick = torch.randperm(pairs.shape[0], generator=gen, device="cuda")[:count].sort().values
    return pos, quat, pairs[pick].to(torch.int32).contiguous(), float(np.float32(state.L)), gen


def _packed(layers):
    return torch.tensor(np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in layers]), device="cuda")


def _model(case, layers):
    sysd = SYSTEMS[case["system"]]
    dims = [layers[0][0].shape[1]] + [W.shape[0] for W, _ in layers]
    device = torch.device("cuda", torch.cuda.current_device())
    return PairModel(sysd["shape"], Hypers(*sysd["hypers"]), dims, sysd["act"], device)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "forces":
        return dict(case=case, system=_system(case, seed))
    if kind == "nlist":
        state = _state(case, case["n"], seed)
        c = _counts(case)
        r, L = c["shape"].cutoff + SKIN, float(np.float32(state.L))
        cap = int(1.3 * c["pairs"](state.N, r)) + 1024
        return dict(case=case, pos=torch.tensor(state.pos, device="cuda"), L=L, r=r, cap=cap,
                    pairs=torch.zeros(cap, 2, dtype=torch.int32, device="cuda"),
                    count=torch.zeros(1, dtype=torch.int64, device="cuda"),
                    ws=torch.empty(size_query("amlp_nlist_workspace_bytes", state.N, L, r), dtype=torch.uint8,
                                   device="cuda"))
    if kind == "run":
        s = _system(case, seed)
        return dict(case=case, system=s, start=s.snapshot_tensors())
    if kind == "pool":
        sysd = SYSTEMS[case["system"]]
        net = EnergyNet(_layers(case, seed), sysd["act"], "cuda")
        pool = NativePool(sysd["shape"], Hypers(*sysd["hypers"]), net, dt=0.005)
        # sizes spread by a factor of four around n
        sizes = [max(500, int(case["n"] * 2.0 ** (2.0 * k / max(1, case["count"] - 1) - 1.0)))
                 for k in range(case["count"])]
        return dict(case=case, net=net, pool=pool,
                    requests=[_state(case, n, seed + 1000 * k) for k, n in enumerate(sizes)])
    layers = _layers(case, seed)
    model = _model(case, layers)
    w = _packed(layers)
    if kind == "vjp":
        pos, quat, pairs, L, gen = _pair_inputs(case, case["pairs"], seed)
        up = torch.rand(pairs.shape[0], generator=gen, device="cuda") + 0.5
        return dict(case=case, model=model, w=w.requires_grad_(), pos=pos.requires_grad_(),
                    quat=quat.requires_grad_(), pairs=pairs, L=L, up=up)
    pos, quat, pairs, L, gen = _pair_inputs(case, case["rows"], seed)
    g = model.descriptors(pos, quat, pairs, L)
    y = torch.rand(g.shape[0], generator=gen, device="cuda")
    return dict(case=case, model=model, w=w, g=g, y=y)


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forces":
        s = state["system"]
        s.compute_forces(case["method"])
        # the energy is a sum of single-precision pair energies, kept in a double
        pe = s.th[Thermostat.pe.offset:Thermostat.pe.offset + 8].view(torch.float64)
        return dict(F=s.F, T=s.T, pe=pe.float())
    if kind == "nlist":
        pos, ws = state["pos"], state["ws"]
        call("amlp_nlist_build", pos.data_ptr(), pos.shape[0], state["L"], state["r"], state["pairs"].data_ptr(),
             state["cap"], state["count"].data_ptr(), ws.data_ptr(), ws.numel(),
             torch.cuda.current_stream().cuda_stream)
        return dict(count=state["count"], pairs=state["pairs"])
    if kind == "run":
        s = state["system"]
        s.restore_tensors(state["start"])
        s.run(RUN_STEPS, "adjoint")
        return dict(pos=s.pos, quat=s.quat, vel=s.vel, angmom=s.angmom)
    if kind == "pool":
        pool = state["pool"]
        ids = [pool.admit(r, kT=1.0) for r in state["requests"]]
        pool.step_segment(POOL_STEPS)
        out = [pool.evict(i) for i in ids]
        return [{k: o[k] for k in ("pos", "quat", "vel", "angmom")} for o in out]
    if kind == "vjp":
        pos, quat, w = state["pos"], state["quat"], state["w"]
        E = pair_energies(pos, quat, w, state["pairs"], state["L"], state["model"])
        g = torch.autograd.grad(E, (pos, quat, w), state["up"])
        return dict(E=E.detach(), pos=g[0], quat=g[1], w=g[2])
    loss, grad = mse_loss_grad(state["model"], state["w"], state["g"], state["y"])
    return dict(loss=loss.float(), grad=grad)


# ------------------------------------------------------------------ least work
def _counts(case):
    sysd = SYSTEMS[case["system"]]
    shape = get_shape(sysd["shape"])
    nr, na, lm = sysd["hypers"][0] + 1, sysd["hypers"][1] + 1, sysd["hypers"][2]
    D = nr + na * lm
    dims = [D] + list(sysd["widths"]) + [1]
    nd = 2 * shape.npts
    # one descriptor: the cheaper of the harmonic form and the sum over unordered point pairs
    k = lm * (lm + 2)
    harmonic = nd * (2 * na * k + 141) + 2 * na * k
    direct = nd * (nd - 1) // 2 * (2 * na * lm + na + 4 * lm + 5) + 75 * nd
    f_net = 2 * sum(dims[i] * dims[i + 1] for i in range(len(dims) - 1))
    rho = sysd.get("rho") or sysd["phi"] / shape.volume
    pairs = lambda n, r: n * 2 / 3 * math.pi * rho * r ** 3  # noqa: E731
    return dict(D=D, dims=dims, f_desc=min(harmonic, direct), f_net=f_net, shape=shape, pairs=pairs,
                weights=sum(dims[i + 1] * (dims[i] + 1) for i in range(len(dims) - 1)))


def work(case):
    c, kind = _counts(case), case["kind"]
    if kind in ("forces", "run", "pool"):
        sizes = [case["n"]]
        if kind == "pool":
            sizes = [max(500, int(case["n"] * 2.0 ** (2.0 * k / max(1, case["count"] - 1) - 1.0)))
                     for k in range(case["count"])]
        n = sum(sizes)
        p, pv = c["pairs"](n, c["shape"].cutoff), c["pairs"](n, c["shape"].cutoff + SKIN)
        per_pair = 10 * (c["f_desc"] + c["f_net"]) if case.get("method", "adjoint") != "adjoint" else \
            3 * c["f_desc"] + 2 * c["f_net"]
        # Verlet pairs in; positions and orientations in, forces and torques out
        step = dict(bytes=8 * pv + n * (12 + 16 + 12 + 12) + 4 * c["weights"], flops=p * per_pair + 12 * pv)
        if kind == "forces":
            return step
        steps = RUN_STEPS if kind == "run" else POOL_STEPS
        # each step also reads and writes the state (positions, orientations, velocities, momenta ...)
        return dict(bytes=steps * (step["bytes"] + 200 * n), flops=steps * (step["flops"] + 500 * n))
    if kind == "nlist":
        pv = c["pairs"](case["n"], c["shape"].cutoff + SKIN)
        return dict(bytes=12 * case["n"] + 8 * pv, flops=10 * pv)
    if kind == "vjp":
        p = case["pairs"]
        return dict(bytes=p * (8 + 4 + 4) + 8 * c["weights"], flops=p * (3 * c["f_desc"] + 3 * c["f_net"]))
    return dict(bytes=4 * case["rows"] * (c["D"] + 1) + 8 * c["weights"], flops=3 * case["rows"] * c["f_net"])


# ------------------------------------------------------------------ 64-bit values
_ACT = {"relu": torch.relu, "tanh": torch.tanh, "silu": torch.nn.functional.silu}


def _descriptor64(p, hypers, rc):
    """The descriptor of clouds p (P, Nd, 3), as NepDescriptorKernels.py:3-144 defines it."""
    nr, na, lm = hypers[0] + 1, hypers[1] + 1, hypers[2]
    r = p - p.mean(dim=1, keepdim=True)
    d = r.square().sum(-1).sqrt()
    u = d / rc
    x = 2 * (u - 1).square() - 1
    fc = 0.5 * (1 + torch.cos(math.pi * u))
    T = [torch.ones_like(x), x]
    while len(T) < nr:
        T.append(2 * x * T[-1] - T[-2])
    f = torch.stack([0.5 * (1 + t) * fc for t in T], 1)
    rh = r / d[..., None]
    c = rh @ rh.transpose(1, 2)
    leg, fa, ang = [torch.ones_like(c), c], f[:, :na], []
    for l in range(1, lm + 1):
        if l > 1:
            leg.append(((2 * l - 1) * c * leg[-1] - (l - 1) * leg[-2]) / l)
        ang.append(((fa @ leg[l]) * fa).sum(-1))
    return torch.cat([f.sum(-1), torch.stack(ang, -1).flatten(1)], 1)


def _net64(g, layers, act):
    for k, (W, b) in enumerate(layers):
        g = torch.nn.functional.linear(g, W, b)
        if k + 1 < len(layers):
            g = _ACT[act](g)
    return g[:, 0]


def _rotate64(q, b):
    """Body points b (K, 3) in the frames of the quaternions q (R, 4), w first: (R, K, 3)."""
    w, x, y, z = q.unbind(1)
    a = w * w - (x * x + y * y + z * z)
    m = torch.stack([a + 2 * x * x, 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), a + 2 * y * y, 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), a + 2 * z * z], 1).view(-1, 3, 3)
    return torch.einsum("rij,kj->rki", m, b)


def _pairs64(case, pos, quat, pairs, L, layers, up=None, clip=True, weight_grads=False, torque=True):
    """Energies of the pairs and the sums over bodies of their forces and torques (weighted by
    ``up``), by automatic differentiation in 64 bits; the weights' gradient too when asked."""
    sysd = SYSTEMS[case["system"]]
    shape = get_shape(sysd["shape"])
    body = torch.tensor(shape.pts, device="cuda").double()
    h = shape.npts
    en_min, en_range = float(shape.en_min), float(shape.en_max) - float(shape.en_min)
    layers = [(torch.tensor(W, device="cuda").double().requires_grad_(weight_grads),
               torch.tensor(b, device="cuda").double().requires_grad_(weight_grads)) for W, b in layers]
    pos, quat = pos.detach().double(), quat.detach().double()
    F, T = torch.zeros_like(pos), torch.zeros_like(pos)
    E, gw = [], [torch.zeros_like(t) for l in layers for t in l]
    step = max(256, 24_000_000 // (2 * h) ** 2)
    for a in range(0, pairs.shape[0], step):
        i, j = pairs[a:a + step].long().unbind(1)
        t = pos[j] - pos[i]
        t = torch.where(t > L / 2, t - L, t)
        t = torch.where(t < -L / 2, t + L, t)[:, None]
        pi, pj = _rotate64(quat[i], body), _rotate64(quat[j], body)
        p = torch.cat([pi, pj + t], 1).requires_grad_(torque)
        e = en_min + en_range * _net64(_descriptor64(p, sysd["hypers"], float(shape.nep_cutoff)), layers, sysd["act"])
        E.append(e.detach())
        want = ([p] if torque else []) + ([t_ for l in layers for t_ in l] if weight_grads else [])
        if not want:
            continue
        s = e.sum() if up is None else (e * up[a:a + step].double()).sum()
        got = torch.autograd.grad(s, want)
        if weight_grads:
            gw = [x + y for x, y in zip(gw, got[-len(gw):])]
        if not torque:
            continue
        g = got[0]
        f = -g[:, :h].sum(1)
        ti = -torch.linalg.cross(pi, g[:, :h]).sum(1)
        tj = -torch.linalg.cross(pj, g[:, h:]).sum(1)
        if clip:
            f, ti, tj = (v.clamp(-100, 100) for v in (f, ti, tj))
        F.index_add_(0, i, f).index_add_(0, j, -f)
        T.index_add_(0, i, ti).index_add_(0, j, tj)
    return torch.cat(E), F, T, torch.cat([x.reshape(-1) for x in gw])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "pool", "nlist"):
        return None  # trajectories and whole numbers
    sysd = SYSTEMS[case["system"]]
    layers = _layers(case, seed)
    if kind == "forces":
        state = _state(case, case["n"], seed)
        pos = torch.tensor(state.pos, device="cuda")
        quat = torch.tensor(state.orient, device="cuda")
        pairs = _pairs_within(pos, state.L, get_shape(sysd["shape"]).cutoff)
        analytic = case["method"] == "adjoint"
        E, F, T, _ = _pairs64(case, pos, quat, pairs, float(np.float32(state.L)), layers, torque=analytic)
        # forward differences of single-precision energies over 1e-5 are mostly rounding: no
        # 64-bit value stands for them
        return dict(F=F if analytic else None, T=T if analytic else None, pe=E.sum().reshape(1))
    if kind == "vjp":
        pos, quat, pairs, L, gen = _pair_inputs(case, case["pairs"], seed)
        up = torch.rand(pairs.shape[0], generator=gen, device="cuda") + 0.5
        E, F, T, gw = _pairs64(case, pos, quat, pairs, L, layers, up=up, clip=False, weight_grads=True)
        w, u = quat.double()[:, :1], quat.double()[:, 1:]
        gq = torch.cat([2 * (T * u).sum(1, keepdim=True), -2 * (w * T + torch.linalg.cross(T, u))], 1)
        return dict(E=E, pos=-F, quat=gq, w=gw)
    s = prepare(case, seed)  # the batch itself is an input
    g, y = s["g"].double(), s["y"].double()
    layers = [(torch.tensor(W, device="cuda").double().requires_grad_(),
               torch.tensor(b, device="cuda").double().requires_grad_()) for W, b in layers]
    loss = (_net64(g, layers, sysd["act"]) - y).square().mean()
    grads = torch.autograd.grad(loss, [t for l in layers for t in l])
    return dict(loss=loss.detach().reshape(1), grad=torch.cat([x.reshape(-1) for x in grads]))
