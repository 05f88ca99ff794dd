"""RKF45 with a CTA per warp-block (bia_pair_block_rkf_kernel, csrc/bia_step.cu) against the ensemble's kernel,
a warp per warp-block: the same sums in the same order, so bitwise the same step and the same
counters, at ragged sizes, with and without charges."""
import numpy as np
import pytest

from bia_3d_gpu_b200 import METHOD_RKF, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charged", [False, True])
@pytest.mark.parametrize("n", [2, 17, 31, 32, 33, 64, 65, 257, 1000])
def test_block_kernel_equals_warp_kernel(cuda, n, charged):
    if charged:
        s, eps, q = initial.coulomb_cube(n, seed=71, dmin=min(1e-2, 0.1 * n ** (-1.0 / 3.0)))
        q = cuda.tensor(q, device="cuda")
    else:
        (s, eps), q = initial.gravity_ball(n=n, seed=71), None
    cfg = default_config(eps_th=eps, dt=1e-5, method=METHOD_RKF)
    with BIASolver() as solver:
        a, b, c = (cuda.tensor(s, device="cuda") for _ in range(3))
        sa = solver.step(a, cfg, q=q)
        ens = solver.ensemble([n], [eps])
        sb = ens.run(b, cfg, 1, q=q)
        cfg.deterministic = 0
        sc = solver.step(c, cfg, q=q)
    assert cuda.equal(a, b) and sa == sb and sa == sc
    # another order of at most n terms a sum
    move = float((a.cpu() - cuda.tensor(s)).abs().max())
    assert float((c - a).abs().max()) <= n * 2.3e-16 * (np.abs(s).max() + n * move)
