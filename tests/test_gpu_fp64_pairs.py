"""GPU: the FP64 form's pair terms and opening test against the oracle, at ordinary and
at extreme distances (where r^3 leaves the exponent range), plain and damped, and with
nodes exactly at the opening radius (a lattice), which take the reference's own test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("scale,mass_scale", [(1.0, 1e11), (1e3, 1e11), (1e115, 1e240), (1e115, 1e100)])
@pytest.mark.parametrize("n", [3, 40, 700])
def test_fp64_forces_over_scales(nb, orc, n, scale, mass_scale, damp):
    rng = np.random.default_rng(n)
    pos, mass = rng.normal(size=(n, 3)) * scale, rng.uniform(1, 2, n) * mass_scale
    with nb.Engine(precision=nb.PRECISION_FP64) as e:
        acc, cnt = e.barnes_hut(pos, mass, damping=damp, counts=True)
    ref, want = orc.forces(pos, mass, 0.5, damping=damp)
    assert np.array_equal(cnt, want)
    # mass times position overflows at (1e115, 1e240): the reference's centres of mass are not finite
    fine = np.isfinite(ref).all(1)
    assert np.array_equal(fine, np.isfinite(acc).all(1))
    assert (np.linalg.norm(acc - ref, axis=1) <= 1e-12 * np.linalg.norm(ref, axis=1))[fine].all()


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("theta", [0.25, 0.5, 1.0])
def test_opening_ties_on_a_lattice(nb, orc, single, theta):
    """Distances that are powers of two times the cell sides: side / distance == theta
    happens, and is not open."""
    g = np.arange(8.0)
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) * 2.0 - 7.0
    mass = np.full(len(pos), 2.0 ** 36)
    with nb.Engine(precision=nb.PRECISION_FP64, datatype_bytes=4 if single else 8) as e:
        _, cnt = e.barnes_hut(pos, mass, theta=theta, counts=True)
    _, want = orc.forces(pos, mass, theta, single=single)
    assert np.array_equal(cnt, want)
