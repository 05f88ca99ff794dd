"""The walk of the universal and learned steps depends on the particles' relative states alone: a velocity common
to all leaves every pair sum bitwise as it is.  Velocities in multiples of 2^-28 and common ones that are
multiples of 2^-10, so that every boosted velocity and every difference is exact."""
import numpy as np
import pytest

from bia_3d_gpu_b200 import METHOD_LEARNED, METHOD_UNIVERSAL, BIASolver, default_config, initial

pytestmark = pytest.mark.gpu


# one warp-block, a CTA per warp-block, a warp per warp-block
@pytest.mark.parametrize("n", [2, 33, 257, 1332])
@pytest.mark.parametrize("method", [METHOD_UNIVERSAL, METHOD_LEARNED])
@pytest.mark.parametrize("charged,dt", [(False, 1e-4), (False, 1e-2), (True, 1e-5)])
def test_common_velocity_leaves_the_pair_sums(cuda, n, method, charged, dt):
    if charged:
        s, eps, q = initial.coulomb_cube(n, seed=91, dmin=min(1e-2, 0.1 * n ** (-1.0 / 3.0)))
        q = cuda.tensor(q, device="cuda")
    else:
        (s, eps), q = initial.plummer(n, seed=91), None
    s[3:] = np.round(s[3:] * 2.0**28) / 2.0**28
    boosted = s.copy()
    boosted[3:] += np.array([[8192.0 + 2.0**-10], [-12345.625], [3000.0]])
    assert np.array_equal(boosted[3:, :1] - boosted[3:], s[3:, :1] - s[3:])
    cfg = default_config(eps_th=eps, dt=dt, method=method)
    sums = []
    with BIASolver() as solver:
        solver.load_heads()
        for state in (s, boosted):
            out = cuda.zeros((6, n), dtype=cuda.float64, device="cuda")
            solver.step_shard(cuda.tensor(state, device="cuda"), cfg, 0, 1, out, q=q)
            sums.append(out.cpu().numpy())
    assert np.abs(sums[0]).max() > 0 and np.array_equal(sums[0], sums[1])
