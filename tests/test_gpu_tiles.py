"""Pair counts at the edges of the force kernels' tiles.

The fused adjoint kernel works on tiles of 128 pairs and the wide path's
descriptor kernels on tiles of 64; both hand each pair to two threads. Counts
just below, at and above one and two tiles, and a single pair, against FP64
autograd of the same pairs, at the contract's 1e-3 (relative, norm over bodies;
for the single pair 2e-3 of its largest component, at least 1).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HYPERS = (10, 8, 4)


def _state(shape_name, seed):
    from amlp.configs import make_state
    from oracle import nep, nlist
    from oracle.shapes import SHAPES
    s = make_state(120, shape_name, 0.35, seed=seed)
    vp = nlist.sorted_pairs(nlist.reference_pairs(s.pos, s.L, 4.5))
    _, pairs, _ = nep.min_image_filter(s.pos, vp, s.L, SHAPES[shape_name]["cutoff"], np.float32)
    return s, pairs


@pytest.mark.parametrize("count", [1, 63, 64, 65, 127, 128, 129, 193])
@pytest.mark.parametrize("shape_name,widths,act,method", [
    ("cube26", (64, 64), "tanh", "amlp_forces_adjoint"),
    ("cyl24", (128, 128), "silu", "amlp_forces_adjoint_wide"),
])
def test_adjoint_forces_at_tile_edges(shape_name, widths, act, method, count):
    import gpu_helpers as H
    from amlp.engine import EnergyNet
    from oracle import adjoint
    from oracle.shapes import SHAPES
    s, pairs = _state(shape_name, seed=11)
    assert len(pairs) >= count
    pairs = pairs[:count]
    layers = EnergyNet.xavier(47, widths, act, seed=5, device="cpu").layers
    F, T, pe = H.fused_forces(s.pos, s.orient, s.L, pairs, SHAPES[shape_name], HYPERS, layers, act, method=method)
    ex = adjoint.exact_pair_forces(s.pos, s.orient, pairs, s.L, SHAPES[shape_name], HYPERS, layers, act)
    for got, ref in ((F, ex["forces"]), (T, ex["torques"])):
        if count == 1:
            np.testing.assert_allclose(got, ref, rtol=0, atol=2e-3 * max(1.0, np.abs(ref).max()))
        else:
            assert np.linalg.norm(got - ref) <= 1e-3 * np.linalg.norm(ref)
    assert abs(pe - ex["E"].sum()) <= 1e-4 * max(1.0, np.abs(ex["E"]).sum())
