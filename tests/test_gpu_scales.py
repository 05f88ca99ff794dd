"""Units: lengths times 2^a and velocities times 2^b (couplings times 2^(a + 2 b), steps times 2^(a - b)) scale
the pair sums by 2^a and 2^b, out to where the squares of the pairs' separations, velocities and angular
momenta leave the type's range.

ALG: a pair's end state is off by roundings of its start and its path, |r| + |g| dt, 64 of them, in
velocity of |g| and of its change.  Universal variables and the learned form: of its displacement,
as tests/test_gpu_pair_sums.py derives it (2e-14, with a learned pair 1e-13)."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_ALG, METHOD_LEARNED, METHOD_UNIVERSAL, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu

N = 6


def pair_sizes(s, eps, dt):
    """(2, N) sums over partners of |r| + |g| dt and |g| + |dg|, and of the displacements' norms."""
    path, disp = np.zeros((2, N)), np.zeros((2, N))
    for i in range(N):
        for j in range(N):
            if i != j:
                r, g = s[:3, i] - s[:3, j], s[3:, i] - s[3:, j]
                h, _ = oracle.pair_halfdisp(r, g, eps, dt, method=METHOD_UNIVERSAL)
                dg = 2 * np.linalg.norm(h[3:])
                path[:, i] += np.linalg.norm(r) + (np.linalg.norm(g) + dg) * dt, np.linalg.norm(g) + dg
                disp[:, i] += np.linalg.norm(h[:3]), dg / 2
    return path, disp


def pair_sums(cuda, method, s, eps, dt, q=None):
    with BIASolver() as solver:
        solver.load_heads()
        out = cuda.zeros(s.shape, dtype=cuda.float64, device="cuda")
        qt = None if q is None else cuda.tensor(q, device="cuda")
        st = solver.step_shard(cuda.tensor(s, device="cuda"), default_config(eps_th=eps, dt=dt, method=method), 0, 1, out,
                               q=qt, stats=True)
        assert st["nonfinite"] == 0, st
        return out.cpu().numpy()


# the ends: a fourth power of a length (2^256), a cube of a velocity (2^341), a squared step (2^512), the
# coupling times the squared step, a length cubed (2^-341), squares near the type's smallest normal number
SCALES = [(-480, 0), (-400, -300), (-400, -100), (-300, -200), (-300, 100), (-200, 400), (-100, -400), (0, 480),
          (200, 200), (400, -100), (480, -300)]
# a step's many pericentre times: the universal variable's cube (step over length) leaves the range there
UV_LONG = [(-200, 400), (-100, -400), (0, 480)]


@pytest.mark.parametrize("method", [METHOD_ALG, METHOD_UNIVERSAL, METHOD_LEARNED])
@pytest.mark.parametrize("dt", [2e-5, 2e-2])
@pytest.mark.parametrize("eps", [-0.05, -20.0, 5.0])  # hyperbolae, mostly ellipses, repulsion
def test_powers_of_two(cuda, method, dt, eps):
    s, _ = initial.plummer(N, seed=9)
    path, disp = pair_sizes(s, eps, dt)
    tol = 2 * (64 * 1.1e-16 * path if method == METHOD_ALG else (1e-13 if method == METHOD_LEARNED else 2e-14) * disp)
    want = pair_sums(cuda, method, s, eps, dt)
    for a, b in SCALES:
        if method != METHOD_ALG and dt > 1e-3 and (a, b) in UV_LONG:
            continue
        unit = 2.0 ** np.array([a, a, a, b, b, b])[:, None]
        got = pair_sums(cuda, method, s * unit, float(np.ldexp(eps, a + 2 * b)), float(np.ldexp(dt, a - b))) / unit
        err = np.linalg.norm((got - want).reshape(2, 3, N), axis=1)
        assert np.all(err <= tol), (a, b, (err / tol).max(1))


@pytest.mark.parametrize("method", [METHOD_UNIVERSAL, METHOD_LEARNED])
@pytest.mark.parametrize("n", [N, 1332])  # a CTA and a warp per warp-block
def test_scaled_charges(cuda, method, n):
    """Couplings eps q_i q_j as they are, their factors far apart: with eps dt^2, or that times a charge, below the
    type's range, and with charges of very different size, zero among them.  2 ulp more for the products' order."""
    s, _ = initial.plummer(n, seed=9)
    rng = np.random.default_rng(4)
    q = 2.0 ** rng.integers(-1, 2, n)
    q[1] = 0.0
    eps, dt = -0.05, 2e-5
    want = pair_sums(cuda, method, s, eps, dt, q)
    size = np.abs(want).max(1, keepdims=True)
    for a in (-500, -480, -400, 400, 450, 500):
        got = pair_sums(cuda, method, s, float(np.ldexp(eps, -2 * a)), dt, np.ldexp(q, a))
        assert np.all(np.abs(got - want) <= (2e-14 + n * 2.3e-16) * size), a
    # lengths about 2^-340, where eps dt^2 q_i q_j is just above the type's smallest normal number or below
    # (the coupling itself, about 2^(a + 2 b), is normal)
    for a, b, k in ((-330, -330, 0), (-345, -200, 0), (-345, -200, 60), (-345, -200, -120), (-300, -100, -200),
                    (-400, -300, -30)):
        unit = 2.0 ** np.array([a, a, a, b, b, b])[:, None]
        e = float(np.ldexp(eps, a + 2 * b - 2 * k))
        assert np.ldexp(e, 2 * k - a - 2 * b) == eps  # exact
        got = pair_sums(cuda, method, s * unit, e, float(np.ldexp(dt, a - b)), np.ldexp(q, k)) / unit
        assert np.all(np.abs(got - want) <= (2e-14 + n * 2.3e-16) * size), (a, b, k)
