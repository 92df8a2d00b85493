"""GPU: an octree that its build reports as malformed is not walked. More than eight
particles at one point overflow the child list of the deepest cell (the build reports
it, beside the coincidence), for the one-block build, the general one and ensembles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,same", [(100, 9), (1000, 70), (5000, 20), (60000, 100)])
def test_malformed_octree_is_not_walked(nb, precision, n, same):
    pos, vel, mass = nb.generate(n, gen_type=1, seed=n)
    bad = pos.copy()
    bad[:same] = bad[0]
    with nb.Engine(precision=precision) as e:
        for systems in (1, 2):
            if systems == 2:
                e.set_systems([n - 3, 3])
            for p in (bad, pos):
                e.set_particles(p, vel, mass)
                if p is bad:
                    with pytest.raises(nb.NBodyError) as err:
                        e.step(2)
                    assert err.value.status == nb.ERR_COINCIDENT
                    assert e.stats()["interactions_total"] == 0
                else:
                    e.step(2)  # the context stays usable
                    assert e.stats()["interactions_total"] > 0
                    assert np.isfinite(e.get_particles()[0]).all()


def test_a_coincident_pair_is_still_walked(nb):
    pos, vel, mass = nb.generate(5000, gen_type=1, seed=1)
    pos[1] = pos[0]
    with nb.Engine() as e:
        with pytest.raises(nb.NBodyError) as err:
            e.barnes_hut(pos, mass)
        assert err.value.status == nb.ERR_COINCIDENT
        assert e.stats()["interactions"] > 0
