"""GPU: the MIXED adjoint's packed pair terms against the FP64 form's, at sizes whose
lists end inside a chunk of eight (and inside a pair), without and with damping, for
groups walked by teams and by single warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damping", [0, 1])
@pytest.mark.parametrize("n", [2, 3, 7, 8, 9, 10, 31, 33, 161, 1001, 6001, 80001])
def test_mixed_adjoint_matches_fp64(nb, n, damping):
    """A term's offset is exact to 2 u Pm (u = 2^-24, Pm the group's extent), a body
    nearer than 2^-9 Pm to the group's box is taken in FP64, and a term changes five
    times as fast as its offset: 5 * 2 u * 2^9 = 3e-4 for the worst pair; three times
    that for sums in which the largest terms partly cancel."""
    pos, _, mass = nb.generate(n, gen_type=1, seed=n, size=64.0)
    la = np.random.default_rng(n).normal(size=pos.shape)
    out = []
    for precision in (0, 1):
        with nb.Engine(precision=precision, damping=damping, theta=0.5) as e:
            out.append(e.force_vjp(pos, mass, la))
    for got, want in zip(*out):
        assert np.isfinite(got).all()
        assert np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want)
