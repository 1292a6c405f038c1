"""The fused finite-difference kernel over body sizes.

Up to 30 points per body it reads the rotated halves of variants 4..9 from
shared memory, above it rotates each point where it is used, as the descriptor
kernel of the separate path does. All ten variants' energies against that path
(descriptors, then the net): descriptors and hidden layers are the same sums in the
same order, and the output layer adds its 64 terms w a, |a| <= 1, and the bias in
another one, so that two energies differ by at most 2 * 65 * 2^-24 (|b| + sum |w|).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HYPERS = (10, 8, 4)


@pytest.mark.parametrize("npts,count", [(7, 33), (8, 1), (26, 32), (29, 65), (30, 31), (31, 33), (31, 64)])
def test_variant_energies_over_cloud_sizes(npts, count):
    import gpu_helpers as gh
    from amlp.configs import make_state
    from amlp.engine import EnergyNet
    from oracle import nlist
    from oracle.shapes import SHAPES
    rng = np.random.default_rng(npts)
    pts = rng.normal(size=(npts, 3))
    pts *= 0.5 / np.linalg.norm(pts, axis=1, keepdims=True)
    shape = dict(SHAPES["cube26"], pts=pts.astype(np.float32))
    s = make_state(120, "cube26", 0.45, seed=5)
    pairs = nlist.sorted_pairs(nlist.reference_pairs(s.pos, s.L, 2.2))
    assert len(pairs) >= count
    pairs = pairs[:count]
    layers = EnergyNet.xavier(47, (64, 64), "tanh", seed=3, device="cpu").layers
    e = gh.fused_forces(s.pos, s.orient, s.L, pairs, shape, HYPERS, layers, "tanh",
                        method="amlp_forces_fd_energies")[3].astype(np.float64)
    ref = gh.mlp_energy(layers, "tanh", gh.descriptors(s.pos, s.orient, s.L, pairs, shape, HYPERS)).astype(np.float64)
    assert e.shape == ref.shape and np.isfinite(e).all()
    W, b = layers[-1]
    assert np.abs(e - ref).max() <= 2 * 65 * 2.0 ** -24 * float(np.abs(W).sum() + np.abs(b).sum())
