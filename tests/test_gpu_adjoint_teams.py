"""GPU: the adjoint particle by particle. Groups walked by teams of warps and by single
warps give the same gradients up to the order of the FP64 sums at the nodes, and the
MIXED form's agree with the FP64 form's for all but a few particles far better than in
the norm of the whole gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(nb, n):
    pos, _, mass = nb.generate(n, gen_type=1, seed=n, size=64.0)
    return pos, mass, np.random.default_rng(n).normal(size=pos.shape)


def errors(got, want):
    """Per particle, relative to its gradient (to the median one where that is larger)."""
    d = np.abs(got - want) if got.ndim == 1 else np.linalg.norm(got - want, axis=1)
    s = np.abs(want) if want.ndim == 1 else np.linalg.norm(want, axis=1)
    return d / np.maximum(s, np.median(s))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("damping", [0, 1])
@pytest.mark.parametrize("n", [161, 2048, 6001])
def test_teams_and_single_warps_give_the_same_gradients(nb, n, damping, precision):
    """A system of its own is walked by teams, beside many single particles by single
    warps. Both sum the same batches in the same order; only the atomics on the nodes
    come in any order: 1e-16 of sums of up to thousands of terms, 1e-10 with cancellation."""
    pos, mass, la = state(nb, n)
    extra = n // 128 + 2  # fewer than 160 particles a system
    with nb.Engine(precision=precision, damping=damping, theta=0.5) as e:
        own = e.force_vjp(pos, mass, la)
        e.set_systems([n] + [1] * extra)
        both = e.force_vjp(np.concatenate([pos, np.arange(3.0 * extra).reshape(-1, 3)]),
                           np.concatenate([mass, np.ones(extra)]), np.concatenate([la, np.zeros((extra, 3))]))
    for got, want in zip(both, own):
        assert errors(got[:n], want).max() <= 1e-10
        assert (got[n:] == 0.0).all()


@pytest.mark.parametrize("damping", [0, 1])
@pytest.mark.parametrize("n", [161, 1001, 6001, 80001])
def test_mixed_adjoint_of_most_particles(nb, n, damping):
    """A term's offset is exact to 2 u Pm (u = 2^-24, Pm the group's extent) and a term
    changes five times as fast: 1e-5 for bodies at Pm / 16, nearer than most particles'
    nearest ones, and 6e-5 at Pm / 100."""
    pos, mass, la = state(nb, n)
    out = []
    for precision in (0, 1):
        with nb.Engine(precision=precision, damping=damping, theta=0.5) as e:
            out.append(e.force_vjp(pos, mass, la))
    for got, want in zip(*out):
        err = errors(got, want)
        assert np.median(err) <= 1e-5 and np.percentile(err, 99) <= 1e-4
