"""GPU: groups walked by teams of warps and by single warps give the same sums bit for
bit, and the reference's counts, also where the queue of waiting nodes is long (a
small theta) and where the last group is ragged. A system of its own with few groups
is walked by teams; the same system inside a large ensemble is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,theta", [(2, 0.5), (159, 0.5), (161, 0.5), (1000, 0.5), (6001, 0.5), (6000, 0.05), (3000, 1e-9)])
def test_team_equals_single_warp_and_reference(nb, orc, precision, n, theta):
    pos, vel, mass = nb.generate(n, gen_type=1, seed=n)
    fill = [nb.generate(3000, gen_type=0, seed=k) for k in range(38)]  # more groups than teams take
    with nb.Engine(precision=precision, theta=theta) as e:
        acc, cnt = e.barnes_hut(pos, mass, theta=theta, counts=True)
        e.set_systems([n] + [3000] * len(fill))
        e.set_particles(np.concatenate([pos] + [f[0] for f in fill]), None, np.concatenate([mass] + [f[2] for f in fill]))
        if theta >= 0.5:
            e.compute_forces()
            assert np.array_equal(e.get_particles(acc=True)[2][:n], acc)
    ref, want = orc.forces(pos, mass, theta)
    assert np.array_equal(cnt, want)
    err = np.linalg.norm(acc - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.percentile(err, 99) <= (1e-12 if precision else 1e-5)


@pytest.mark.parametrize("precision", [0, 1])
def test_team_equals_single_warp_with_a_long_queue(nb, precision):
    """theta = 0.05: thousands of waiting nodes, so the newest go first for a while."""
    parts = [nb.generate(3000, gen_type=1, seed=k) for k in range(39)]
    with nb.Engine(precision=precision, theta=0.05) as e:
        own = e.barnes_hut(parts[0][0], parts[0][2], theta=0.05)
        e.set_systems([3000] * len(parts))
        e.set_particles(np.concatenate([p[0] for p in parts]), None, np.concatenate([p[2] for p in parts]))
        e.compute_forces()
        assert np.array_equal(e.get_particles(acc=True)[2][:3000], own)


@pytest.mark.parametrize("precision,n", [(0, 56832), (0, 56833), (1, 113664), (1, 113665), (1, 131072), (1, 131073)])
def test_counts_on_both_sides_of_the_size_limits(nb, orc, precision, n):
    """Teams end at 56,832 (MIXED) and 113,664 (FP64) particles, the mass pass's groups
    of lanes per node at 131,072."""
    pos, vel, mass = nb.generate(n, gen_type=2, size=1024.0, seed=n)
    sample = np.sort(np.random.default_rng(n).choice(n, 300, replace=False)).astype(np.uint32)
    sample[-1] = n - 1
    with nb.Engine(precision=precision) as e:
        acc, cnt = e.barnes_hut(pos, mass, counts=True)
    ref, want = orc.forces(pos, mass, 0.5, sample=sample)
    assert np.array_equal(cnt[sample], want)
    err = np.linalg.norm(acc[sample] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.percentile(err, 99) <= (1e-12 if precision else 1e-5)
