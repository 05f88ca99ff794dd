"""The ALG conic pairs at the places where the solvers branch (hyperbola and ellipse, csrc/bia_pair.cuh): starts
at pericentre, apocentre and next to them, either sense of rotation, circular orbits, attractive and
repulsive hyperbolae, far out on an asymptote, steps from far below an orbit's time (the Taylor and
reversion starts) to several orbits (the reference's guess), exact parabolae.  Each pair alone, against the
same algorithm in quad precision to 1e-12 of its size: four ulps times at most 1e3, the separation over the
pericentre scale, that the angle's rounding is magnified by."""
import math

import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_ALG, BIASolver, default_config

pytestmark = pytest.mark.gpu


def _orbit(e, nu, mu, p, sense, rng):
    """Relative state of semi-latus rectum p at true anomaly nu, in a random plane."""
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    r = p / (1.0 + e * math.cos(nu))
    pos = r * (math.cos(nu) * q[0] + math.sin(nu) * q[1])
    vel = math.sqrt(abs(mu) / p) * (-math.sin(nu) * q[0] + (e + math.cos(nu)) * q[1])
    return pos, sense * vel


def _check(cuda, pos, vel, eps, dt, cls):
    s = np.zeros((6, 2))
    s[:3, 0], s[3:, 0] = pos, vel
    ref, _, _ = oracle.bia_step(s, eps, dt, quad=True)
    t = cuda.tensor(s, device="cuda")
    with BIASolver() as solver:
        st = solver.step(t, default_config(eps_th=eps, dt=dt, method=METHOD_ALG))
    got = t.cpu().numpy()
    assert st[cls] == 1 and st["nonfinite"] == 0, st
    size, speed = max(np.abs(ref[:3]).max(), np.abs(s[:3]).max()), max(np.abs(ref[3:]).max(), np.abs(s[3:]).max())
    assert np.abs(got[:3] - ref[:3]).max() <= 1e-12 * size
    assert np.abs(got[3:] - ref[3:]).max() <= 1e-12 * speed


@pytest.mark.parametrize("e", [0.0, 1e-3, 0.4, 0.9])
@pytest.mark.parametrize("nu", [0.0, 1e-9, 1.0, -2.0, math.pi, math.pi - 1e-7])
@pytest.mark.parametrize("frac", [1e-7, 1e-3, 4e-3, 0.3, 2.6])
def test_ellipses(cuda, e, nu, frac):
    rng = np.random.default_rng(int(1e3 * e) + int(10 * abs(nu)))
    mu, p = 0.7, 1.3
    period = 2 * math.pi * math.sqrt((p / (1 - e * e)) ** 3 / mu)
    for sense in (1.0, -1.0):
        pos, vel = _orbit(e, nu, mu, p, sense, rng)
        _check(cuda, pos, vel, -mu, frac * period, "ellipse")


@pytest.mark.parametrize("e", [1.2, 3.0, 40.0])
@pytest.mark.parametrize("where", [0.0, 1e-9, 0.3, -0.8, 0.97, -0.97])
@pytest.mark.parametrize("frac", [1e-7, 1e-4, 2e-3, 0.5, 20.0])
@pytest.mark.parametrize("repulsive", [False, True])
def test_hyperbolae(cuda, e, where, frac, repulsive):
    rng = np.random.default_rng(int(10 * e) + int(100 * abs(where)))
    mu, p = 0.7, 1.3
    # the other branch of the same conic is the repulsive orbit: r = p / (e cos nu - 1)
    span = math.acos((1.0 if repulsive else -1.0) / e)
    nu = where * span
    for sense in (1.0, -1.0):
        if repulsive:
            q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
            r = p / (e * math.cos(nu) - 1.0)
            pos = r * (math.cos(nu) * q[0] + math.sin(nu) * q[1])
            vel = sense * math.sqrt(mu / p) * (-math.sin(nu) * q[0] + (math.cos(nu) - e) * q[1]) * -1.0
            eps = mu
        else:
            pos, vel = _orbit(e, nu, mu, p, sense, rng)
            r, eps = np.linalg.norm(pos), -mu
        _check(cuda, pos, vel, eps, frac * r / np.linalg.norm(vel), "hyperbola")


@pytest.mark.parametrize("dt", [1e-3, 0.5])
def test_exact_parabola_keeps_its_branch(cuda, dt):
    # |g|^2 = 2 / r exactly: 1 = 2 / 2
    _check(cuda, np.array([2.0, 0.0, 0.0]), np.array([0.0, 1.0, 0.0]), -1.0, dt, "parabola")
