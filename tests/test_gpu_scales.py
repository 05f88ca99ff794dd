"""Units: lengths times 2^a and velocities times 2^b (couplings times 2^(a + 2 b), steps times 2^(a - b)) scale
the pair sums by 2^a and 2^b, out to where the squares of the pairs' separations, velocities and angular
momenta leave the type's range.

ALG: a pair's end state is off by roundings of its start and its path, |r| + |g| dt, 64 of them, in
velocity of |g| and of its change."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_ALG, METHOD_UNIVERSAL, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu

N = 6


def pair_sizes(s, eps, dt):
    """(2, N) sums over partners of |r| + |g| dt and |g| + |dg|."""
    path = np.zeros((2, N))
    for i in range(N):
        for j in range(N):
            if i != j:
                r, g = s[:3, i] - s[:3, j], s[3:, i] - s[3:, j]
                h, _ = oracle.pair_halfdisp(r, g, eps, dt, method=METHOD_UNIVERSAL)
                dg = 2 * np.linalg.norm(h[3:])
                path[:, i] += np.linalg.norm(r) + (np.linalg.norm(g) + dg) * dt, np.linalg.norm(g) + dg
    return path


def pair_sums(cuda, method, s, eps, dt):
    with BIASolver() as solver:
        out = cuda.zeros(s.shape, dtype=cuda.float64, device="cuda")
        st = solver.step_shard(cuda.tensor(s, device="cuda"), default_config(eps_th=eps, dt=dt, method=method), 0, 1, out,
                               stats=True)
        assert st["nonfinite"] == 0, st
        return out.cpu().numpy()


# the ends: a fourth power of a length (2^256), a cube of a velocity (2^341), a squared step (2^512), the
# coupling times the squared step, a length cubed (2^-341), squares near the type's smallest normal number
SCALES = [(-480, 0), (-400, -300), (-400, -100), (-300, -200), (-300, 100), (-200, 400), (-100, -400), (0, 480),
          (200, 200), (400, -100), (480, -300)]


@pytest.mark.parametrize("method", [METHOD_ALG])
@pytest.mark.parametrize("dt", [2e-5, 2e-2])
@pytest.mark.parametrize("eps", [-0.05, -20.0, 5.0])  # hyperbolae, mostly ellipses, repulsion
def test_powers_of_two(cuda, method, dt, eps):
    s, _ = initial.plummer(N, seed=9)
    path = pair_sizes(s, eps, dt)
    tol = 2 * 64 * 1.1e-16 * path
    want = pair_sums(cuda, method, s, eps, dt)
    for a, b in SCALES:
        unit = 2.0 ** np.array([a, a, a, b, b, b])[:, None]
        got = pair_sums(cuda, method, s * unit, float(np.ldexp(eps, a + 2 * b)), float(np.ldexp(dt, a - b))) / unit
        err = np.linalg.norm((got - want).reshape(2, 3, N), axis=1)
        assert np.all(err <= tol), (a, b, (err / tol).max(1))
