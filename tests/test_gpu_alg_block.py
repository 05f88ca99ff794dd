"""ALG with a CTA per warp-block (bia_pair_block_kernel, csrc/bia_step.cu) against the phase-locked
kernel: the same sums in the same order, so bitwise the same step and the same counters, at ragged
sizes, on both sides of the lines where the default changes kernels, for hyperbolic, elliptic and
mixed systems with and without charges."""
import numpy as np
import pytest

from bia_3d_gpu_b200 import METHOD_ALG, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu


def system(kind, n):
    if kind == "coulomb":
        s, eps, q = initial.coulomb_cube(n, seed=61, dmin=min(1e-3, 0.1 * n ** (-1.0 / 3.0)))
        return s, eps, q, 1e-5
    s, eps = (initial.cold_ball if kind == "cold" else initial.gravity_ball)(n=n, seed=61)
    s = np.array(s)
    if kind == "mixed":  # a third of the particles at rest: ellipses among the hyperbolae
        s[3:, ::3] *= 1e-3
        s[:, 5::7] = s[:, 4:-1:7][:, : s[:, 5::7].shape[1]] + 1e-4  # close pairs
    return s, eps, None, 1e-4


@pytest.mark.parametrize("kind", ["ball", "cold", "mixed", "coulomb"])
@pytest.mark.parametrize("n", [2, 17, 31, 32, 33, 64, 65, 257, 1000])
def test_block_kernel_equals_phase_kernel(cuda, kind, n):
    s, eps, q, dt = system(kind, n)
    qt = None if q is None else cuda.tensor(q, device="cuda")
    cfg = default_config(eps_th=eps, dt=dt, method=METHOD_ALG)
    outs = []
    with BIASolver() as solver:
        for shape in ("tiles8", "phase32", None):
            solver.set_shape(METHOD_ALG, n, shape)
            t = cuda.tensor(s, device="cuda")
            outs.append((solver.step(t, cfg, q=qt), t.cpu().numpy()))
        cfg.deterministic = 0
        t = cuda.tensor(s, device="cuda")
        st = solver.step(t, cfg, q=qt)
    for o in outs[1:]:
        assert np.array_equal(o[1], outs[0][1], equal_nan=True) and o[0] == outs[0][0]
    assert st == outs[0][0]
    # another order of at most n terms a sum
    move = np.abs(outs[0][1] - s).max()
    assert np.abs(t.cpu().numpy() - outs[0][1]).max() <= n * 2.3e-16 * (np.abs(s).max() + n * move)


@pytest.mark.parametrize("n", [2656, 2657, 3072, 3105, 3780, 3810])
def test_default_is_bitwise_the_same_across_its_lines(cuda, n):
    s, eps, q, dt = system("coulomb", n)
    qt = cuda.tensor(q, device="cuda")
    cfg = default_config(eps_th=eps, dt=dt, method=METHOD_ALG)
    outs = []
    with BIASolver() as solver:
        for shape in (None, "tiles8", "phase32_lane"):
            solver.set_shape(METHOD_ALG, n, shape)
            t = cuda.tensor(s, device="cuda")
            outs.append((solver.step(t, cfg, q=qt), t.cpu().numpy()))
    for o in outs[1:]:
        assert np.array_equal(o[1], outs[0][1]) and o[0] == outs[0][0]
