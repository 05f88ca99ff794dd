"""The universal and learned steps with a CTA per warp-block (bia_pair_walk_block_kernel, csrc/bia_step.cu)
against the ensemble's walk, a warp per warp-block: the same sums in the same order, so bitwise the same
step and the same counters, at ragged sizes, on both sides of the line, with and without charges, for
short steps, steps where most pairs leave the short-step series, and a backward step (none take it)."""
import numpy as np
import pytest

from bia_3d_gpu_b200 import METHOD_LEARNED, METHOD_UNIVERSAL, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [METHOD_UNIVERSAL, METHOD_LEARNED])
@pytest.mark.parametrize("charged,dt", [(False, 1e-4), (False, 1e-2), (True, 1e-5), (True, 1e-4), (False, -1e-4)])
@pytest.mark.parametrize("n", [2, 17, 31, 32, 33, 64, 65, 257, 736, 737])
def test_block_kernel_equals_walk(cuda, method, charged, dt, n):
    if charged:
        s, eps, q = initial.coulomb_cube(n, seed=81, dmin=min(1e-2, 0.1 * n ** (-1.0 / 3.0)))
        q = cuda.tensor(q, device="cuda")
    else:
        (s, eps), q = initial.plummer(n, seed=81), None
    cfg = default_config(eps_th=eps, dt=dt, method=method)
    with BIASolver() as solver:
        solver.load_heads()
        a, b, c = (cuda.tensor(s, device="cuda") for _ in range(3))
        sa = solver.step(a, cfg, q=q)
        sb = solver.ensemble([n], [eps]).run(b, cfg, 1, q=q)
        cfg.deterministic = 0
        sc = solver.step(c, cfg, q=q)
    assert cuda.equal(a, b) and sa == sb and sa == sc
    # another order of at most n terms a sum
    move = float((a.cpu() - cuda.tensor(s)).abs().max())
    assert float((c - a).abs().max()) <= n * 2.3e-16 * (np.abs(s).max() + n * move)
