"""GPU: the walk's block shape where teams of warps walk the groups: what the statistics
report, and that tuning such a state does not choose the shape of single warps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_statistics_report_the_teams(nb):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n, team in ((100, False), (5000, True), (50001, True)):
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
    limit = 12 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
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
