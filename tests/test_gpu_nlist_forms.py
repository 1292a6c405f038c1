"""The Verlet build's forms against the pair criterion itself, pair by pair.

Below 9,472 bodies a warp takes one body, from there on four that share a
traversal when they share a cell; lists of up to 128 later neighbours are ranked
by counting, longer ones by a bitonic network; bodies outside the box switch the
FP32 pre-test from shifted cell columns to folded components. The lists must equal
the FP64 criterion's (scipy's where its input checks allow it) exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _brute(pos, L, r):
    """All pairs i < j by the FP64 criterion: float32(pos + L/2) in a box of edge
    float32(L + 1e-4), folded once per axis, compared inclusively."""
    x = (np.asarray(pos, np.float32) + np.float32(np.float32(L) * np.float32(0.5))).astype(np.float64)
    fb = float(np.float32(L) + np.float32(0.0001))
    out = []
    for i in range(len(x)):
        d = x[i] - x[i + 1:]
        d = np.where(d < -0.5 * fb, fb + d, np.where(d > 0.5 * fb, d - fb, d))
        d = d * d
        j = np.nonzero((d[:, 0] + d[:, 1]) + d[:, 2] <= r * r)[0] + i + 1
        out.append(np.stack([np.full(len(j), i), j], 1))
    return np.concatenate(out)


@pytest.mark.parametrize("n", [9471, 9472, 9473, 9476])
def test_one_and_four_bodies_per_warp(n):
    import gpu_helpers as H
    from oracle import nlist
    L = np.float32(33.0)
    pos = (np.random.default_rng(n).random((n, 3)) * L - L / 2).astype(np.float32)
    got, count = H.nlist(pos, L, 4.5)
    ref = nlist.sorted_pairs(nlist.reference_pairs(pos, L, 4.5))
    assert count == len(ref) and np.array_equal(got, ref)


@pytest.mark.parametrize("n,L", [(200, 20.0), (1500, 14.0), (1500, 10.5), (3000, 14.0)])
def test_bodies_outside_the_box_and_dense_lists(n, L):
    import gpu_helpers as H
    rng = np.random.default_rng(n)
    L = np.float32(L)
    pos = (rng.random((n, 3)) * L - L / 2).astype(np.float32)
    for shift in (0.0, 0.05):  # every body inside; some of them out by up to 0.05
        p = pos + np.float32(shift) * rng.uniform(-1, 1, (n, 3)).astype(np.float32)
        got, count = H.nlist(p, L, 4.5)
        ref = _brute(p, L, 4.5)
        assert count == len(ref) and np.array_equal(got, ref)


def test_pairs_near_the_radius():
    """Distances within a few FP32 roundings of r, across the faces too."""
    import gpu_helpers as H
    rng = np.random.default_rng(3)
    L, r, m = np.float32(40.0), 4.5, 1500
    a = (rng.random((m, 3)) * L - L / 2).astype(np.float32)
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    b = a + u * (r * (1 + rng.normal(0, 3e-7, (m, 1))))
    b = (b + L / 2) % float(L) - L / 2
    pos = np.concatenate([a, b]).astype(np.float32)
    pos = np.clip(pos, -L / 2, np.nextafter(L / 2, np.float32(0)))
    got, count = H.nlist(pos, L, r)
    ref = _brute(pos, L, r)
    assert count == len(ref) and np.array_equal(got, ref)
