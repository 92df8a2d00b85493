"""GPU: the FP64 all-pairs sums at the edges of their tiles (targets per warp and
block, sources per chunk) against the oracle's compensated direct sum. Both sum
exactly up to a few roundings of each pair term, so 1e-13 of the result's size
leaves two orders of magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (33, 7), (1000, 1), (8192, 9), (8193, 8), (20000, 17)])
def test_direct_forces_at_tile_edges(nb, orc, n, m, damp):
    pos, vel, mass = nb.generate(n, gen_type=1, seed=n)
    targets = np.random.default_rng(m).choice(n, m, replace=False).astype(np.uint32)
    targets[-1] = targets[0]  # a target may be asked for twice
    want = orc.direct(pos, mass, targets=targets, damping=damp)
    with nb.Engine() as e:
        e.set_particles(pos, vel, mass)
        got = e.direct_forces(targets, damping=damp)
    scale = np.maximum(np.linalg.norm(want, axis=1), 1e-300)
    assert (np.linalg.norm(got - want, axis=1) / scale).max() <= 1e-13


def test_direct_forces_over_extreme_distances(nb):
    """Pairs whose r^3 leaves the exponent range take the plain formula."""
    pos = np.array([[0.0, 0.0, 0.0], [1e-105, 0.0, 0.0], [0.0, 1e120, 0.0]])
    mass = np.array([1e-190, 1e-200, 1e300])
    with nb.Engine() as e:
        e.set_particles(pos, np.zeros_like(pos), mass)
        got = e.direct_forces()
    G = 6.67384e-11
    assert np.isclose(got[0, 0], mass[1] * G / 1e-105 / 1e-105, rtol=1e-13)
    assert np.isclose(got[1, 0], -mass[0] * G / 1e-105 / 1e-105, rtol=1e-13)
    assert np.isclose(got[0, 1], mass[2] * G / 1e120 / 1e120, rtol=1e-13)
