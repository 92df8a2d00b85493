"""GPU: collision pairs against a brute-force search in numpy, at the edges of the
search's groups and stack. With a vanishing theta every node is opened, so every
pair within range collides; dt = 0 leaves the merged particles where the merge put
them (components folded in ascending index, src/main.cpp:423-430)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def merged(pos, vel, mass, rng):
    n = len(mass)
    d = np.sqrt(((pos[:, None] - pos[None]) ** 2).sum(-1))
    label = np.arange(n)
    for _ in range(n):  # smallest index reachable within range
        near = np.where(d < rng, label[None], n).min(1)
        if np.array_equal(near, label):
            break
        label = np.minimum(near, label[near])
    out = []
    for r in range(n):
        if label[r] != r:
            continue
        p, v, m = pos[r].copy(), vel[r].copy(), mass[r]
        for k in range(r + 1, n):
            if label[k] == r:
                p = (p * m + pos[k] * mass[k]) / (m + mass[k])
                v = (v * m + vel[k] * mass[k]) / (m + mass[k])
                m = m + mass[k]
        out.append((*p, *v, m))
    return np.array(out)


@pytest.mark.parametrize("n,rng", [(2, 1.0), (2, 1e-3), (31, 5.0), (33, 5.0), (64, 1e4), (700, 3.0), (700, 12.0), (700, 1e4)])
@pytest.mark.parametrize("clusters", [1, 2])
def test_collisions_equal_brute_force(nb, n, rng, clusters):
    g = np.random.default_rng(n)
    pos = g.uniform(-0.5, 0.5, (n, 3)) * (2.0 if n == 2 and rng < 1 else 0.5 if n == 2 else 60.0)
    if clusters == 2:
        pos[::2] += 5000.0  # groups that straddle the root's halves
    vel, mass = g.normal(size=(n, 3)), g.uniform(5e10, 5e11, n)
    want = merged(pos, vel, mass, rng)
    with nb.Engine(precision=nb.PRECISION_FP64, theta=1e-9, dt=0.0, collide=1, collision_range=rng) as e:
        e.set_particles(pos, vel, mass)
        e.step(1)
        p, v = e.get_particles()
        m = e.get_masses()
    got = np.concatenate([p, v, m[:, None]], 1)
    assert got.shape == want.shape
    assert np.allclose(got, want, rtol=1e-12, atol=1e-9)
