"""GPU: the one-block build of small systems against the general build (the same
particles as the first of two systems, which are always built by the general kernels)
and the reference's counts: block and warp edges, both datatypes, keys that need the
second and the third word, and what is reported as coincident or not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def states(nb, n, kind):
    pos, vel, mass = nb.generate(n, gen_type=1, seed=n)
    if kind == "second word" and n > 3:  # a cluster that shares the first word, two far particles
        pos *= 1e-2
        pos[0] = [1e7, 3.0, -2.0]
        pos[1] = [-1e7, -5.0, 7.0]
    elif kind == "third word" and n > 2:  # pairs closer than 2^-42 of the root
        pos[1] = pos[0] + 1e-11
        pos[n // 2] = pos[n - 1] - 1e-11
    elif kind == "zero mass":
        mass[:] = 0.0
    return pos, vel, mass


@pytest.mark.parametrize("datatype_bytes", [8, 4])
@pytest.mark.parametrize("kind", ["plain", "second word", "third word", "zero mass"])
@pytest.mark.parametrize("n", [2, 3, 32, 33, 64, 65, 511, 1023, 1024, 1025])
def test_small_build_equals_general_build(nb, orc, n, kind, datatype_bytes):
    pos, vel, mass = states(nb, n, kind)
    if datatype_bytes == 4 and kind == "third word":
        pytest.skip("the pairs coincide in float")
    with nb.Engine(precision=nb.PRECISION_FP64, datatype_bytes=datatype_bytes) as e:
        acc, cnt = e.barnes_hut(pos, mass, counts=True)
        st = e.stats()
        e.set_systems([n, 2])
        e.set_particles(np.concatenate([pos, [[0.0, 0, 0], [1.0, 2, 3]]]), None, np.concatenate([mass, [1.0, 2.0]]))
        e.compute_forces()
        assert np.array_equal(e.get_particles(acc=True)[2][:n], acc, equal_nan=True)
        assert e.stats()["tree_depth"] >= st["tree_depth"]
    assert (st["sort_passes"] == 0) == (n <= 1024)
    _, want = orc.forces(pos, mass, 0.5, single=datatype_bytes == 4)
    assert np.array_equal(cnt, want)


@pytest.mark.parametrize("n", [5, 700])
def test_small_build_reports_bad_input(nb, n):
    pos, vel, mass = nb.generate(n, seed=n)
    with nb.Engine() as e:
        for what in ("pos", "mass", "same"):
            p, m = pos.copy(), mass.copy()
            if what == "pos":
                p[n // 2, 1] = np.nan
            elif what == "mass":
                m[n - 1] = np.inf
            else:
                p[n - 1] = p[0]
            with pytest.raises(nb.NBodyError) as err:
                e.barnes_hut(p, m)
            assert err.value.status == (nb.ERR_COINCIDENT if what == "same" else nb.ERR_NONFINITE)
        assert np.isfinite(e.barnes_hut(pos, mass)).all()  # the context stays usable


def test_small_build_adaptive_steps(nb, orc):
    """max |v| of the one-block build drives the adaptive step."""
    pos, vel, mass = nb.generate(300, gen_type=1, seed=4)
    vel = vel + 50.0
    with nb.Engine(precision=nb.PRECISION_FP64, adaptive=1, max_vel_change=1e9, max_pos_change=0.5, dt=0.0333,
                   min_adaptive_dt=1e-6) as e:
        e.set_particles(pos, vel, mass)
        e.step(1)
        assert np.isclose(e.stats()["last_dt"], 0.5 / np.linalg.norm(vel, axis=1).max(), rtol=1e-14)
