"""The pair sums themselves (without the drift, whose size hides them in a whole step), positions and velocities
apart, against the pairs' half-displacements in quad precision, relative to the interaction.

The universal and learned walk: a pair's f - 1 and f' carry a handful of FP64 roundings (2^-53 = 1.1e-16
each) on top of those of r0^-3 (about ten), g - dt and g' - 1 less: 5e-15 of |h| a pair is more than
40 roundings.  The sum of m terms adds m roundings of the sum of magnitudes.  Pairs that leave the short-step
series (a few at the longer steps, a close one among them) solve for the root with Stumpff functions after up to
three duplications (4^3 x 1.1e-16, and the rest): 2e-14.  A learned pair ends with a Halley step whose accepted residual
leaves 1e-13 at most."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_ALG, METHOD_LEARNED, METHOD_RKF, METHOD_UNIVERSAL, BIASolver, default_config
from bia_3d_gpu_b200 import find_dxyuv_kernel, initial

pytestmark = pytest.mark.gpu


def quad_sums(s, eps, dt, q, method):
    """(6, n) sums over partners of the half-displacements, and of their norms (2, n)."""
    n = s.shape[1]
    h = np.zeros((6, n, n))
    for i in range(n):
        for j in range(i + 1, n):
            e = eps if q is None else eps * q[i] * q[j]
            h[:, i, j], _ = oracle.pair_halfdisp(s[:3, i] - s[:3, j], s[3:, i] - s[3:, j], e, dt, method=method, quad=True)
            h[:, j, i] = -h[:, i, j]
    size = np.linalg.norm(h.reshape(2, 3, n, n), axis=1).sum(2)
    return h.sum(2), size


@pytest.mark.parametrize("n", [2, 33, 64])
@pytest.mark.parametrize("dt", [1e-5, 2e-4, 1e-3])
@pytest.mark.parametrize("charged", [False, True])
def test_walk_pair_sums(cuda, n, dt, charged):
    if charged:
        s, eps, q = initial.coulomb_cube(n, seed=n, dmin=0.02)
        dt = dt * 0.1
    else:
        (s, eps), q = initial.plummer(n, seed=n), None
    want, size = quad_sums(s, eps, dt, q, METHOD_UNIVERSAL)
    assert size.min() > 0
    qt = None if q is None else cuda.tensor(q, device="cuda")
    with BIASolver() as solver:
        solver.load_heads()
        for method, deterministic in ((METHOD_UNIVERSAL, 1), (METHOD_UNIVERSAL, 0), (METHOD_LEARNED, 1)):
            cfg = default_config(eps_th=eps, dt=dt, method=method)
            cfg.deterministic = deterministic
            out = cuda.zeros((6, n), dtype=cuda.float64, device="cuda")
            st = solver.step_shard(cuda.tensor(s, device="cuda"), cfg, 0, 1, out, q=qt, stats=True)
            got = out.cpu().numpy()
            learned = st["hyperbola"] + st["ellipse"]
            pair = 1e-13 if learned else 2e-14 if st["iter_universal"] else 5e-15
            err = np.linalg.norm((got - want).reshape(2, 3, n), axis=1)
            assert np.all(err <= (pair + n * 1.2e-16) * size), (method, deterministic, (err / size).max(1), st)


@pytest.mark.parametrize("method", [METHOD_RKF, METHOD_ALG])
@pytest.mark.parametrize("n", [2, 34, 66])
def test_row_displacements(cuda, method, n):
    """The drop-in row at a step so long that a pair's displacement is far above what its solver's end leaves.
    Both solvers form the end state in the pair's plane, so a pair is off by roundings of the
    start and of the path, |r| + |g| dt (64 of them), and in velocity of |g|; RKF45 besides by its
    tolerance of 1e-16 a step, over at most thirty steps."""
    s, eps = initial.plummer(70, seed=51)
    s = np.ascontiguousarray(s[:, :n])
    dt = 0.2
    acc = np.zeros((6, n))
    rel = np.ascontiguousarray((s[:, :1] - s).T).reshape(-1)
    out = np.full(6 * n, np.nan)
    assert find_dxyuv_kernel(method, n, 1, eps, dt, 18, *acc, rel, out) == 0
    h = out.reshape(n, 6).T
    for j in range(1, n):
        r, g = s[:3, 0] - s[:3, j], s[3:, 0] - s[3:, j]
        want, _ = oracle.pair_halfdisp(r, g, eps, dt, method=METHOD_UNIVERSAL, quad=True)
        path = np.linalg.norm(r) + np.linalg.norm(g) * dt
        extra = 30 * 1e-16 if method == METHOD_RKF else 0.0
        for part, scale in ((slice(0, 3), path), (slice(3, 6), np.linalg.norm(g) + 2 * np.linalg.norm(want[3:]))):
            tol = 64 * 1.1e-16 * scale + extra
            assert np.linalg.norm(want[part]) > 1e4 * tol
            assert np.linalg.norm(h[part, j] - want[part]) <= tol, (j, part)
