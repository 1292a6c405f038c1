"""The net pass of the wide force path at the edges of its rounds.

A round is two tiles of 128 rows for each of 148 blocks; the last one may leave
a block with one tile, or with none. Row counts on both sides of one tile, of
148 and of 296 tiles, for nets whose two operand tiles fit shared memory, whose
first one lies in tensor memory, and that run one tile at a time, against FP64
autograd at the contract's 1e-3 (relative, norm over bodies). The list is a short
one repeated, so that the exact result is a multiple of the short list's. For
ReLU it holds the pairs whose pre-activations are clear of the kink by 1e-3: a
derivative that jumps there is not the rounding's to decide.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HYPERS = (10, 8, 4)
SHAPE = "cyl24"


def _pairs(layers, act):
    from amlp.configs import make_state
    from oracle import adjoint, nep, nlist
    from oracle.shapes import SHAPES
    s = make_state(120, SHAPE, 0.35, seed=11)
    vp = nlist.sorted_pairs(nlist.reference_pairs(s.pos, s.L, 4.5))
    pairs = nep.min_image_filter(s.pos, vp, s.L, SHAPES[SHAPE]["cutoff"], np.float32)[1]
    if act == "relu":
        pairs = pairs[adjoint.relu_margin(s.pos, s.orient, pairs, s.L, SHAPES[SHAPE], HYPERS, layers) > 1e-3]
    return s, pairs


@pytest.mark.parametrize("count", [1, 128, 129, 148 * 128 - 1, 148 * 128 + 1, 296 * 128, 296 * 128 + 1])
@pytest.mark.parametrize("widths,act", [
    ((128, 128), "silu"),             # two tiles in shared memory, act' in tensor memory
    ((64, 80, 48, 64), "relu"),       # two tiles in shared memory
    ((150,), "relu"),                 # one layer: its weights stay
    ((160, 160, 160, 160), "relu"),   # the first tile in tensor memory
    ((96, 96, 96), "tanh"),           # one tile at a time
])
def test_net_pass_at_round_edges(widths, act, count):
    import gpu_helpers as H
    from amlp.engine import EnergyNet
    from oracle import adjoint
    from oracle.shapes import SHAPES
    layers = EnergyNet.xavier(47, widths, act, seed=5, device="cpu").layers
    s, base = _pairs(layers, act)
    assert len(base) > 0
    pairs = np.concatenate([base] * (count // len(base) + 1))[:count]
    F, T, pe = H.fused_forces(s.pos, s.orient, s.L, pairs, SHAPES[SHAPE], HYPERS, layers, act,
                              method="amlp_forces_adjoint_wide")
    full, rest = divmod(count, len(base))
    ref = {"forces": 0.0, "torques": 0.0}
    esum = eabs = 0.0
    for times, part in ((full, base), (1, base[:rest])):
        if times == 0 or len(part) == 0:
            continue
        ex = adjoint.exact_pair_forces(s.pos, s.orient, part, s.L, SHAPES[SHAPE], HYPERS, layers, act)
        for k in ref:
            ref[k] = ref[k] + times * ex[k]
        esum += times * ex["E"].sum()
        eabs += times * np.abs(ex["E"]).sum()
    for got, r in ((F, ref["forces"]), (T, ref["torques"])):
        assert np.linalg.norm(got - r) <= 1e-3 * max(np.linalg.norm(r), 2.0 if count == 1 else 0.0)
    assert abs(pe - esum) <= 1e-4 * max(1.0, eabs)
