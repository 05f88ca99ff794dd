"""The short-step pair of the universal-variable walk (uv_fast_pair, csrc/bia_pair.cuh) and the
walk's queue of other pairs (csrc/bia_uv_walk.cuh).

On the CPU the four series are restated with the kernel's mix of FP64 and FP32 and checked in
extended precision against the solved universal Kepler equation over the region where the kernel
takes them, and the region against the exactness bounds |c_k| <= (3e-4)^k of uv_series.

The tolerances of the series: f - 1 and f' carry h, so three FP64 roundings near 1 (4e-16); g - dt
and g' - 1 multiply contributions of at most |g| dt/(3 r0) <= 1.5e-4 and |g| dt/(2 r0) <= 2.2e-4 of h,
so 1e-13 leaves 2.2e-17 of h.
"""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_LEARNED, METHOD_UNIVERSAL, BIASolver, default_config, initial
from conftest import max_rel_err, rel_err

L = np.longdouble
LIMIT = 1.9e-7


def _region(rng, count):
    """a, b, U with a^2 <= b and b + |U| <= LIMIT, out to its edge."""
    t = np.where(rng.random(count) < 0.5, 1.0 - 1e-9, 10 ** rng.uniform(-6, 0, count)) * LIMIT
    f = np.where(rng.random(count) < 0.2, 1.0, rng.random(count))
    b, U = t * f, t * (1 - f) * np.where(rng.random(count) < 0.7, 1, -1)
    a = np.sqrt(b) * np.where(rng.random(count) < 0.3, 1.0, rng.uniform(-1, 1, count))
    return a, b, U


def test_short_steps_are_exact_by_the_reversion_bounds():
    a, b, U = _region(np.random.default_rng(1), 400_000)
    q = b - U
    y, z, w = a / 2, q / 6, U - q
    c = [y, 2 * y * y - z, y * (5 * z + w / 12 - 5 * y * y),
         y * y * (14 * y * y - 21 * z - w / 2) + z * (3 * z + w / 20)]
    for k in range(4):
        assert np.abs(c[k]).max() <= 3e-4 ** (k + 1), k


def _reference(a, b, U):
    """(f - 1), f', (g - 1), (g' - 1) at dt = r0 = 1 in extended precision, over -U/2, -U, -U/6, -U/2."""
    mu, beta = U, 2 * U - b
    fact = [L(1)]
    for k in range(1, 30):
        fact.append(fact[-1] * k)
    s = L(1) + 0 * U
    for _ in range(30):
        x = beta * s * s
        c = [sum((-x) ** j / fact[2 * j + m] for j in range(8)) for m in range(4)]
        s = s - (s * c[1] + a * s * s * c[2] + mu * s ** 3 * c[3] - 1) / (c[0] + a * s * c[1] + mu * s * s * c[2])
    x = beta * s * s
    c = [sum((-x) ** j / fact[2 * j + m] for j in range(8)) for m in range(4)]
    rt = c[0] + a * s * c[1] + mu * s * s * c[2]
    return 2 * s * s * c[2], s * c[1] / rt, 6 * s ** 3 * c[3], 2 * s * s * c[2] / rt


def test_short_step_series_against_the_solved_equation():
    a, b, U = _region(np.random.default_rng(2), 20_000)
    U = np.where(U == 0, 1e-12, U)
    q = b - U
    f4 = np.float32
    A, Q, V = f4(a), f4(q), f4(U)
    A2 = A * A
    p3 = f4(-0.25) * A * (f4(7) * A2 - f4(3) * Q - V)
    p4 = A2 * (f4(2.625) * A2 - f4(1.75) * Q - f4(7 / 12) * V) + Q * (f4(0.125) * Q + f4(1 / 15) * V) + V * f4(1 / 360) * V
    p45 = p4 - A * p4
    cf, cfd, aU = p3 + p45, f4(2.5) * p3 + f4(3) * p45, A * V
    cg = f4(2 / 3) * p3 - f4(0.25 / 3) * aU + f4(0.1 / 3) * V
    cgd = f4(2) * p3 + f4(2.5) * p4 - f4(0.25) * aU + f4(1 / 12) * V
    p2 = 1.25 * a * a - 0.25 * q - U / 12
    got = [(p2 + cf) - a + 1, 2 * (p2 - 0.75 * a) + cfd + 1, 3 * ((0.6 * p2 + (-0.5 * a + cg)) + 1 / 3),
           2 * ((1.5 * p2 + cgd) - a + 0.5)]
    ref = _reference(L(1) * a, L(1) * b, L(1) * U)
    for g, r, tol in zip(got, ref, (4e-16, 4e-16, 1e-13, 1e-13)):
        assert float(np.abs(g / r - 1).max()) <= tol


# sizes at the edges of the 32-particle blocks; steps where nearly every pair is a short one, where blocks
# hold a few others (the queue) or many (finished on the spot), where the queue is full or just not
@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 161])
@pytest.mark.parametrize("dt", [1e-5, 2e-4, 6e-4, 1e-3, 3e-2, -1e-4])
@pytest.mark.parametrize("charged", [False, True])
def test_walk_matches_oracle(cuda, n, dt, charged):
    if charged:
        s, eps, q = initial.coulomb_cube(n, seed=n, dmin=0.02)
        dt = dt * 0.1
    else:
        s, eps = initial.plummer(n, seed=n)
        q = None
    ref, disp, _ = oracle.bia_step(s, eps, dt, method=METHOD_UNIVERSAL, q=q)
    qt = None if q is None else cuda.tensor(q, device="cuda")
    pairs = n * (n - 1) // 2
    with BIASolver() as solver:
        solver.load_heads()
        for method in (METHOD_UNIVERSAL, METHOD_LEARNED):
            for deterministic in (1, 0):
                cfg = default_config(eps_th=eps, dt=dt, method=method)
                cfg.deterministic = deterministic
                t = cuda.tensor(s, device="cuda")
                d = cuda.zeros_like(t)
                st = solver.step(t, cfg, q=qt, disp=d)
                got = t.cpu().numpy()
                for part in (slice(0, 3), slice(3, 6)):
                    assert rel_err(got[part], ref[part]) <= 1e-12 and max_rel_err(got[part], ref[part]) <= 1e-12
                assert st["universal"] + st["hyperbola"] + st["ellipse"] == pairs and st["nonfinite"] == 0
