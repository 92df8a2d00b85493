"""GPU: the sort statistics of a replayed step are those of its own builds, whatever the
call before it was, and a system built in one block plans no passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def settled(e, pos, vel, mass):
    """Steps until the step is captured and its plan has settled; the plan."""
    for _ in range(6):
        e.set_particles(pos, vel, mass)
        e.step(1)
    return e.stats()["sort_next_passes"]


def test_replay_after_a_small_system(nb):
    pos, vel, mass = nb.generate(5000, gen_type=1, seed=1)
    with nb.Engine() as e:
        plan = settled(e, pos, vel, mass)
        assert plan > 0
        e.barnes_hut(pos[:600], mass[:600])
        st = e.stats()
        assert st["sort_passes"] == 0 and st["sort_next_passes"] == 0
        e.set_particles(pos, vel, mass)
        e.step(1)
        assert e.stats()["sort_passes"] == plan == e.stats()["sort_next_passes"]


def test_replay_of_systems_after_a_single_one(nb):
    counts = [3000, 2000]
    pos, vel, mass = nb.generate(5000, gen_type=1, seed=1)
    deep = pos * 1e-3  # shares the first key word: a full sort
    deep[0], deep[1] = [1e7, 3.0, -2.0], [-1e7, -5.0, 7.0]
    with nb.Engine() as e:
        e.set_systems(counts)
        plan = settled(e, pos, vel, mass)
        assert 0 < plan <= 8
        e.barnes_hut(deep, mass)
        assert e.stats()["sort_passes"] >= 16
        e.set_particles(pos, vel, mass)
        e.step(1)
        assert e.stats()["sort_passes"] == plan == e.stats()["sort_next_passes"]
