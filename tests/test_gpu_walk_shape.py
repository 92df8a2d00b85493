"""GPU: the walk's block shape where teams of warps walk the groups (MIXED: up to ten
groups an SM): what the statistics report, that tuning such a state does not choose the
shape of single warps, and the reference's counts on both sides of the limit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_statistics_report_the_teams(nb):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n, team in ((100, False), (5000, True), (40001, True), (320 * sms, True), (320 * sms + 1, False), (50001, False)):
        pos, vel, mass = nb.generate(n, gen_type=1, seed=1)
        with nb.Engine() as e:
            e.set_particles(pos, vel, mass)
            shape = e.autotune()
            if team:
                assert shape == {"warps_per_block": 4, "blocks": min(-(-n // 32), 5 * sms)}
            else:
                assert shape["blocks"] % sms == 0


def test_a_state_for_single_warps_is_tuned_after_one_for_teams(nb):
    """Both sizes lie in one power of two."""
    limit = 10 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    spent = []
    with nb.Engine(autotune=1) as e:
        for n in (limit - 500, limit + 500):
            pos, vel, mass = nb.generate(n, gen_type=1, seed=1)
            e.set_particles(pos, vel, mass)
            before = e.stats()["kernel_launches"]
            e.step(1)
            spent.append(e.stats()["kernel_launches"] - before)
        assert e.stats()["walk_warps_per_block"] in (1, 2, 4)
    # 3 passes and a step; 3 passes for each of up to 6 shapes and a step
    assert spent[1] > 2 * spent[0]


@pytest.mark.parametrize("more", [0, 1])
def test_counts_on_both_sides_of_the_mixed_limit(nb, orc, more):
    n = 10 * 32 * torch.cuda.get_device_properties(0).multi_processor_count + more
    pos, vel, mass = nb.generate(n, gen_type=2, size=1024.0, seed=n)
    sample = np.sort(np.random.default_rng(n).choice(n, 300, replace=False)).astype(np.uint32)
    sample[-1] = n - 1
    with nb.Engine() as e:
        acc, cnt = e.barnes_hut(pos, mass, counts=True)
        assert (e.stats()["walk_blocks"] == 5 * torch.cuda.get_device_properties(0).multi_processor_count) == (more == 0)
    ref, want = orc.forces(pos, mass, 0.5, sample=sample)
    assert np.array_equal(cnt[sample], want)
    err = np.linalg.norm(acc[sample] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.percentile(err, 99) <= 1e-5


@pytest.mark.parametrize("theta,team", [(0.24, False), (0.25, True), (0.5, True)])
def test_small_opening_angles_end_teams_sooner(nb, theta, team):
    """From seven groups an SM, below 0.25; a call's own angle counts."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 7 * 32 * sms + 1
    pos, vel, mass = nb.generate(n, gen_type=2, size=1024.0, seed=1)
    with nb.Engine() as e:
        e.barnes_hut(pos, mass, theta=theta)
        assert (e.stats()["walk_blocks"] == 5 * sms) == team
        e.barnes_hut(pos[:-1], mass[:-1], theta=theta)
        assert e.stats()["walk_blocks"] == 5 * sms
