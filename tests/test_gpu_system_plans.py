"""GPU: sort plans of several systems. The first build sorts in full (18 passes); later
ones sort the top bits of the system's number and the first key word together, sort
the runs that this leaves tied in place, and fall back to the full sort when a run is
too long. Whatever the plan, the forces stay the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def systems(nb, counts, seed=0):
    parts = [nb.generate(int(n), gen_type=s % 3, size=1024.0 if s % 3 else 512.0, seed=seed + 31 * s)
             for s, n in enumerate(counts)]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[2] for p in parts])


def forces(e, pos, mass):
    e.set_particles(pos, None, mass)
    e.compute_forces()
    return e.get_particles(acc=True)[2], e.stats()


@pytest.mark.parametrize("counts", [[3000, 1], [1, 2, 5000], [40] * 255 + [900], [37] * 257, [9000, 4097, 4096, 4095, 33]])
@pytest.mark.parametrize("datatype_bytes", [8, 4])
def test_planned_sort_of_systems_equals_full_sort(nb, counts, datatype_bytes):
    pos, mass = systems(nb, counts)
    with nb.Engine(precision=nb.PRECISION_FP64, datatype_bytes=datatype_bytes) as e:
        e.set_systems(counts)
        full, st = forces(e, pos, mass)
        assert st["sort_passes"] == 18
        for _ in range(3):
            plan = st["sort_next_passes"]
            acc, st = forces(e, pos, mass)
            assert st["sort_passes"] == plan <= 8
            assert np.array_equal(acc, full)


def test_system_with_a_long_run_takes_the_full_sort(nb):
    """One system becomes a tight cluster with far outliers, whose particles share the
    first key word: a run of thousands, so the full sort follows the planned one."""
    counts = [4000, 6000, 500]
    pos, mass = systems(nb, counts, seed=5)
    tied = pos.copy()
    tied[4000:10000] *= 1e-3
    tied[4000] = [1e7, 3.0, -2.0]
    tied[4001] = [-1e7, -5.0, 7.0]
    with nb.Engine(precision=nb.PRECISION_FP64) as fresh:
        fresh.set_systems(counts)
        want, _ = forces(fresh, tied, mass)
    with nb.Engine(precision=nb.PRECISION_FP64) as e:
        e.set_systems(counts)
        first, st = forces(e, pos, mass)
        plan = st["sort_next_passes"]
        got, st = forces(e, tied, mass)
        assert plan <= 8 and st["sort_passes"] == plan + 18
        assert np.array_equal(got, want)
        again, st = forces(e, tied, mass)
        assert np.array_equal(again, want)
        back, _ = forces(e, pos, mass)
        assert np.array_equal(back, first)


def test_full_sort_over_many_tiles(nb):
    """A single system whose cluster shares the first key word, over several sort tiles."""
    pos, _, mass = nb.generate(70001, gen_type=1, seed=3)
    tied = pos * 1e-3
    tied[0] = [1e7, 3.0, -2.0]
    tied[1] = [-1e7, -5.0, 7.0]
    with nb.Engine() as fresh:
        want, cw = fresh.barnes_hut(tied, mass, counts=True)
    with nb.Engine() as e:
        e.barnes_hut(pos, mass)
        plan = e.stats()["sort_next_passes"]
        got, cg = e.barnes_hut(tied, mass, counts=True)
        assert plan < 8 and e.stats()["sort_passes"] == plan + 16
    assert np.array_equal(got, want) and np.array_equal(cg, cw)
