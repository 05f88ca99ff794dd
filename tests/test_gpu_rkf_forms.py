"""The two forms of the per-pair RKF45 step (rkf_pair, csrc/bia_pair.cuh): reciprocal square roots where
the pair's separation is well inside the type's range, the reference's divisions and roots
elsewhere.  One system scaled by powers of ten over both sides of the rule (positions and
velocities by L, the coupling by L^3, the absolute tolerance by L: the same steps), against the
oracle to 1e-12, with absolute and relative tolerances."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import METHOD_RKF, BIASolver, default_config, initial
from conftest import max_rel_err, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-101, 1e-99, 1.0, 1e60])
@pytest.mark.parametrize("relerr,abserr", [(0.0, 1e-16), (1e-12, 1e-16), (1e-9, 0.0)])
def test_rkf_forms_match_oracle(cuda, scale, relerr, abserr):
    n, dt = 37, 1e-3
    s, eps = initial.gravity_ball(n, seed=17)
    s, eps, abserr = s * scale, eps * scale * scale * scale, abserr * scale
    ref, _, rst = oracle.bia_step(s, eps, dt, method=0, relerr=relerr, abserr=abserr)
    cfg = default_config(eps_th=eps, dt=dt, method=METHOD_RKF, rkf_relerr=relerr, rkf_abserr=abserr)
    t = cuda.tensor(s, device="cuda")
    with BIASolver() as solver:
        st = solver.step(t, cfg)
    got = t.cpu().numpy()
    # scaled back to 1: the norms of numbers beyond 1e154 overflow
    got, ref = got / scale, ref / scale
    for part in (slice(0, 3), slice(3, 6)):
        assert rel_err(got[part], ref[part]) <= 1e-12 and max_rel_err(got[part], ref[part]) <= 1e-12
    # at the small scales |r x g|^2 underflows and the pairs count as degenerate ones; at large ones,
    # beyond 1e76, it overflows and no frame is left to compare
    assert st["rkf"] + st["degenerate"] == n * (n - 1) // 2 and st["nonfinite"] == 0
