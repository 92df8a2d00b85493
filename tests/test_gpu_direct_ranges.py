"""GPU: the FP64 all-pairs sums where G M r^-3 leaves the exponent range and the force does
not, and over more than one launch of targets and more than sixteen chunks of sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 6.67384e-11
U = np.array([3.0, -4.0, 12.0]) / 13.0


def term(d, mass, damping):
    """The reference's pair term, in its order of operations."""
    r2 = (d * d).sum()
    r = np.sqrt(r2)
    return (d / r) * ((mass * G) * (1.0 / (r2 + np.exp(-r)) if damping else 1.0 / r2))


BOTH = [(1e-105, 1e11), (1e-93, 1e40), (1e-93, -1e40), (1e-60, 1e-110), (1e-150, 1.0), (1e60, 1e-100), (1e60, 1e135),
        (1e108, 1e11), (1e110, 1e11), (1.0, 1e-250), (1.0, 1e250), (1e3, 0.0), (1e110, 0.0), (1.0, 1e11)]


@pytest.mark.parametrize("r,m,damping", [(r, m, d) for r, m in BOTH for d in (False, True)] + [(1e-150, 1e200, True)])
def test_forces_whose_cube_leaves_the_range(nb, r, m, damping):
    """A dozen correctly rounded operations (and an exponential of under 2 ulp): 1e-14."""
    pos = np.array([[0.0, 0.0, 0.0], r * U])
    mass = np.array([m, 2.0 * m])
    want = np.array([term(pos[1] - pos[0], mass[1], damping), term(pos[0] - pos[1], mass[0], damping)])
    assert np.isfinite(want).all() and (m == 0.0) == (want == 0.0).all()
    with nb.Engine() as e:
        e.set_particles(pos, np.zeros_like(pos), mass)
        got = e.direct_forces(damping=damping)
    assert np.allclose(got, want, rtol=1e-14, atol=0.0)


def test_ordinary_and_extreme_pairs_in_one_sum(nb):
    """A lane meets both kinds, and both of a warp's targets."""
    rng = np.random.default_rng(0)
    n = 200
    pos, mass = rng.normal(size=(n, 3)), rng.uniform(1e10, 1e11, n)
    pos[::7] *= 1e108
    mass[::5] *= 1e150
    want = np.array([np.sum([term(pos[k] - pos[i], mass[k], False) for k in range(n) if k != i], 0) for i in range(n)])
    size = np.array([np.sum([abs(term(pos[k] - pos[i], mass[k], False)) for k in range(n) if k != i], 0) for i in range(n)])
    with nb.Engine() as e:
        e.set_particles(pos, np.zeros_like(pos), mass)
        got = e.direct_forces()
    assert (np.abs(got - want) <= 1e-13 * size).all()


def test_slabs_of_targets_and_the_most_chunks(nb, orc):
    """65,536 targets a launch; sixteen chunks from 122,881 sources, each larger than
    8192 from 131,073. The tolerance is that of the sums within one launch."""
    n = 131101
    pos, vel, mass = nb.generate(n, gen_type=1, seed=3)
    some = np.array([0, 1, 65534, 65535, 65536, 65537, 131071, 131072, n - 1], dtype=np.uint32)
    want = orc.direct(pos, mass, targets=some)
    scale = np.linalg.norm(want, axis=1)
    with nb.Engine() as e:
        e.set_particles(pos, vel, mass)
        every = e.direct_forces()
        assert every.shape == (n, 3)
        assert (np.linalg.norm(every[some] - want, axis=1) <= 1e-13 * scale).all()
        targets = np.random.default_rng(1).integers(0, n, 65536 + 7).astype(np.uint32)
        targets[[0, 65535, 65536, -1]] = targets[5]
        assert np.array_equal(e.direct_forces(targets), every[targets])
