"""The universal-variable solvers where a reciprocal that they take is not a normal number.

The iteration where an iterate lies so far above the root that F' = r(s) is in the last
factor of four of the type's range, beyond which 1/F' is subnormal: a fly-by that starts at its
pericentre and goes 708 to 710 times as far in the step (the start dt/r0 is then sqrt(-beta) s = 708 to 710,
and F' about r0 e^709 / 2), on both sides of 2^1022, against the same pair in quad precision.

The tolerance: the root (about 7.3) is well conditioned, F and the composition come from Stumpff functions
after five to six duplications, each of which can multiply a relative rounding error by four: 4^6 x 1.1e-16 =
4.5e-13, twice (the root's error and the composition's), and a little for the sums: 2e-12.

The learned pair's Halley step where F'^2 is there, separations of 2^511, among smaller and unscaled ones: what
it accepts is off by 1e-15 at most, the composition as above.  And where the residual times F' is infinite
(lengths of 2^480, velocities of 2^-300): an infinite step is no accepted one."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_LEARNED, METHOD_UNIVERSAL, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [METHOD_UNIVERSAL, METHOD_LEARNED])
@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("ratio", [700.0, 708.9, 709.05, 709.2, 709.4, 709.6, 709.75, 709.85, 710.3])
def test_start_far_above_the_root(cuda, method, sign, ratio):
    r0, v = 0.5, 1.0
    eps = sign * 1e-3 * r0 * v * v
    dt = ratio * r0 / v
    s = np.zeros((6, 2))
    s[0, 0], s[4, 0] = r0, v
    want, _ = oracle.pair_halfdisp(s[:3, 0], s[3:, 0], eps, dt, method=METHOD_UNIVERSAL, quad=True)
    with BIASolver() as solver:
        solver.load_heads()
        t = cuda.tensor(s, device="cuda")
        sums = cuda.zeros((6, 2), dtype=cuda.float64, device="cuda")
        st = solver.step_shard(t, default_config(eps_th=eps, dt=dt, method=method), 0, 1, sums, stats=True)
        got = sums.cpu().numpy()
    assert st["universal"] == 1 and st["nonconverged"] == 0 and st["nonfinite"] == 0
    assert np.array_equal(got[:, 1], -got[:, 0])
    for part in (slice(0, 3), slice(3, 6)):
        assert np.linalg.norm(got[part, 0] - want[part]) <= 2e-12 * np.linalg.norm(want[part])


@pytest.mark.parametrize("scale", [0, 300, 509, 510, 511])
@pytest.mark.parametrize("v", [0.9, 2.2])  # an ellipse, a hyperbola
def test_learned_pair_of_extreme_size(cuda, scale, v):
    r0, v0 = 1.2 * 2.0**scale, v * 2.0**-24
    eps = -(2.0**-48) * r0
    dt = 0.3 * r0 * 2.0**24
    s = np.zeros((6, 2))
    s[0, 0], s[3, 0], s[4, 0] = r0, -0.1 * v0, v0
    want, _ = oracle.pair_halfdisp(s[:3, 0], s[3:, 0], eps, dt, method=METHOD_UNIVERSAL, quad=True)
    with BIASolver() as solver:
        solver.load_heads()
        t = cuda.tensor(s, device="cuda")
        sums = cuda.zeros((6, 2), dtype=cuda.float64, device="cuda")
        st = solver.step_shard(t, default_config(eps_th=eps, dt=dt, method=METHOD_LEARNED), 0, 1, sums, stats=True)
        got = sums.cpu().numpy()
    assert st["nonfinite"] == 0 and st["nonconverged"] == 0
    if scale < 509:
        assert st["learned"] == 1
    for part in (slice(0, 3), slice(3, 6)):
        unit = r0 if part.start == 0 else v0
        assert np.linalg.norm(got[part, 0] / unit - want[part] / unit) <= 2e-12 * np.linalg.norm(want[part] / unit)


@pytest.mark.parametrize("eps", [-0.05, -20.0])
def test_learned_residual_beyond_the_range(cuda, eps):
    s, _ = initial.plummer(6, seed=9)
    sums = []
    with BIASolver() as solver:
        solver.load_heads()
        for a, b in ((0, 0), (480, -300)):
            unit = 2.0 ** np.array([a, a, a, b, b, b])[:, None]
            t = cuda.tensor(s * unit, device="cuda")
            out = cuda.zeros_like(t)
            cfg = default_config(eps_th=float(np.ldexp(eps, a + 2 * b)), dt=float(np.ldexp(2e-2, a - b)), method=METHOD_LEARNED)
            st = solver.step_shard(t, cfg, 0, 1, out, stats=True)
            assert st["nonfinite"] == 0 and st["learned"] > 0
            sums.append(out.cpu().numpy() / unit)
    for part in (slice(0, 3), slice(3, 6)):
        assert np.abs(sums[1][part] - sums[0][part]).max() <= 2e-12 * np.abs(sums[0][part]).max()
