"""GPU: the sort plan of many systems of one or two particles. So few pairs of
neighbours stay tied that the bins alone would shrink the plan below the bits of the
system's number; it has to cover them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[1] * 380 + [2] * 20, [2] * 50 + [1] * 250, [1, 2] * 30 + [1] * 4000,
                                    [1] * 65505 + [2] * 31, [1] * 100 + [2] * 20, [1, 1200]])
def test_plan_covers_the_systems_number(nb, counts):
    n = sum(counts)
    rng = np.random.default_rng(n)
    pos, mass = rng.uniform(-500.0, 500.0, (n, 3)), rng.uniform(1e10, 1e11, n)
    least = -(-(len(counts) - 1).bit_length() // 8)
    with nb.Engine(precision=nb.PRECISION_FP64) as e:
        e.set_systems(counts)
        e.set_particles(pos, None, mass)
        e.compute_forces()
        full = e.get_particles(acc=True)[2]
        assert e.stats()["sort_passes"] == 18
        for _ in range(3):
            plan = e.stats()["sort_next_passes"]
            assert least <= plan <= 8
            e.compute_forces()
            assert e.stats()["sort_passes"] == plan
            assert np.array_equal(e.get_particles(acc=True)[2], full)
    # two particles attract each other along the line between them, one alone feels nothing
    start = np.concatenate([[0], np.cumsum(counts)[:-1]])
    one = start[np.array(counts) == 1]
    assert (full[one] == 0.0).all()
    two = start[np.array(counts) == 2]
    if len(two):
        d = pos[two + 1] - pos[two]
        want = 6.67384e-11 * mass[two + 1, None] * d / np.linalg.norm(d, axis=1)[:, None] ** 3
        assert np.allclose(full[two], want, rtol=1e-13)
