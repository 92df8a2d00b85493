"""GPU: the walk's queue at small opening angles, where it is at its limit for most of the
walk: tiles stay full, teams and single warps keep one order, counts are the reference's,
on ordinary states and on one whose octree is deep and wide at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def nested(n, seed=0):
    """Clusters within clusters: each level's octants hold a part, one the next level."""
    rng = np.random.default_rng(seed)
    scale = 0.25 ** rng.integers(0, 9, n)
    return rng.uniform(-1.0, 1.0, (n, 3)) * scale[:, None] + 0.7 * (1.0 - scale)[:, None], rng.uniform(1e10, 1e11, n)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("theta", [0.02, 0.05, 0.1, 0.3, 0.44, 0.46])
@pytest.mark.parametrize("n", [3000, 20000, 60000])
def test_tiles_stay_full(nb, n, theta, precision):
    """28 of 32 entries on average, beside the dozen tiles of a walk's start and end: a CPU
    model of the queue gives 30 for an octree that is full for six levels, its worst."""
    if n * n / theta > 5e10:
        pytest.skip("long")
    pos, _, mass = nb.generate(n, gen_type=0, size=512.0, seed=n)
    with nb.Engine(precision=precision, theta=theta) as e:
        e.set_walk_stats(True)
        e.set_particles(pos, None, mass)
        e.compute_forces()
        st = e.stats()
    groups = -(-n // 32)
    assert st["walk_tiles"] <= st["walk_entries"] / 28 + 12 * groups
    assert st["max_stack"] <= 2048


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["cube", "nested"])
@pytest.mark.parametrize("n,theta", [(700, 0.1), (5000, 0.02), (5000, 0.3), (5000, 0.449), (5000, 0.45), (24000, 0.1)])
def test_one_order_and_the_reference_counts(nb, orc, n, theta, kind, precision):
    pos, mass = (nested(n) if kind == "nested" else nb.generate(n, gen_type=0, size=512.0, seed=n)[::2])
    with nb.Engine(precision=precision, theta=theta) as e:
        own, cnt = e.barnes_hut(pos, mass, theta=theta, counts=True)
        extra = n // 128 + 2  # fewer than 160 particles a system: single warps
        e.set_systems([n] + [1] * extra)
        e.set_particles(np.concatenate([pos, np.arange(3.0 * extra).reshape(-1, 3)]), None,
                        np.concatenate([mass, np.ones(extra)]))
        e.compute_forces()
        assert np.array_equal(e.get_particles(acc=True)[2][:n], own)
    sample = np.sort(np.random.default_rng(n).choice(n, 200, replace=False)).astype(np.uint32)
    ref, want = orc.forces(pos, mass, theta, sample=sample)
    assert np.array_equal(cnt[sample], want)
    err = np.linalg.norm(own[sample] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.percentile(err, 99) <= (1e-12 if precision else 1e-5)
