"""The resident DIM kernel (dim_resident_kernel, csrc/dim_rkf.cu) at the edges of its shapes: particles per CTA
(n around multiples of the SM count, fewer particles than SMs), tiles (n around 1024), both tracks together
(n <= 4096) or one after the other, the largest sizes it takes (smaller tiles, fewer rows of sums); small
ones against the CPU restatement of rkf_c_ (same accepted steps and derivatives, 1e-12), large ones
against the kernel that keeps its state in global memory (BIA_DIM_COOP_BLOCKS; the same steps, 1e-13)."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import BIASolver, initial, rkf_c
from conftest import max_rel_err, rel_err

pytestmark = pytest.mark.gpu


def _gpu(cuda, s, eps, xe):
    t = cuda.tensor(s, device="cuda")
    with BIASolver() as solver:
        st = solver.dim_integrate(t, eps, 0.0, xe)
        solver.stream.synchronize()
    return t.cpu().numpy(), st


@pytest.mark.parametrize("n", [1, 2, 3, 31, 147, 148, 149, 297, 593])
def test_small_sizes_match_oracle(cuda, n):
    s, eps = initial.gravity_ball(n, seed=100 + n)
    xe = 2e-4
    y0 = np.ascontiguousarray(s.T).reshape(-1)
    yn, ier, nacc, nde = oracle.dim_rkf(y0, eps / 2, 0.0, xe)
    ref = yn.reshape(-1, 6).T
    got, st = _gpu(cuda, s, eps / 2, xe)
    assert ier == 0 and st["ier"] == 0 and st["accepted"] == nacc and st["nde"] == nde
    out = rkf_c(y0.size, eps / 2, 0.0, xe, y0.copy(), 1, 0.0, 1e-16)
    assert out["IER"] == 0 and out["NDE"] == nde
    for g in (got, out["YHN"].reshape(-1, 6).T):
        for part in (slice(0, 3), slice(3, 6)):
            assert rel_err(g[part], ref[part]) <= 1e-12 and max_rel_err(g[part], ref[part]) <= 1e-12


@pytest.mark.parametrize("n", [1023, 1024, 1025, 2049, 4095, 4097, 8191, 20001, 32768])
def test_large_sizes_match_the_global_memory_kernel(cuda, n, monkeypatch):
    s, eps = initial.plummer(n, seed=n)
    xe = 1e-5
    got, st = _gpu(cuda, s, eps / 2, xe)
    monkeypatch.setenv("BIA_DIM_COOP_BLOCKS", "1024")
    ref, rst = _gpu(cuda, s, eps / 2, xe)
    assert st["ier"] == 0 and rst["ier"] == 0
    assert st["accepted"] == rst["accepted"] and st["nde"] == rst["nde"]
    for part in (slice(0, 3), slice(3, 6)):
        assert rel_err(got[part], ref[part]) <= 1e-13 and max_rel_err(got[part], ref[part]) <= 1e-13
