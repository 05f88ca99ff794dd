"""The counters of a walk whose warps solve more than 2^31 pairs each in one launch (bia_uv_walk.cuh): a
universal-variable step with atomic accumulators, so large that 8 warps on 2 CTAs of 148 SMs average
2.2e9 pairs.  About 40 s; every pair is a short-step one."""
import pytest

from bia_3d_gpu_b200 import METHOD_UNIVERSAL, BIASolver, default_config

pytestmark = pytest.mark.gpu


def test_pair_count_beyond_31_bits_a_warp(cuda):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    warps = sms * 2 * 8
    n = int((2 * 2.23e9 * warps) ** 0.5)
    g = cuda.Generator(device="cuda").manual_seed(5)
    s = cuda.zeros((6, n), dtype=cuda.float64, device="cuda")
    s[:3] = cuda.rand((3, n), dtype=cuda.float64, device="cuda", generator=g)
    cfg = default_config(eps_th=-1e-9, dt=1e-6, method=METHOD_UNIVERSAL)
    cfg.deterministic = 0
    with BIASolver() as solver:
        st = solver.step(s, cfg)
    assert st["universal"] == n * (n - 1) // 2
    assert 0 <= st["nonfinite"] == 0 and st["nonconverged"] == 0 and 0 <= st["iter_universal"] <= st["universal"]
