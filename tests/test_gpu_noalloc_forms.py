"""bia_step_noalloc with the kernels that need an opt-in for their shared memory (a CTA per warp-block): RKF45
at every size, universal variables up to two warp-blocks per SM (n = 736 on 148 SMs) and ALG; bitwise the
context's step.  And after the device's primary context was reset, which forgets every opt-in, in
a process of its own: the same calls on new buffers, with and without a new bia_context."""
import ctypes
import os
import subprocess
import sys

import pytest

from bia_3d_gpu_b200 import METHOD_ALG, METHOD_RKF, METHOD_UNIVERSAL, BIASolver, capi, default_config, initial

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("method", [METHOD_ALG, METHOD_RKF, METHOD_UNIVERSAL])
@pytest.mark.parametrize("n", [1, 33, 257, 736, 737, 2048])
def test_noalloc_step_equals_context_step(cuda, method, n):
    s, eps = initial.plummer(n, seed=63)
    cfg = default_config(eps_th=eps, dt=1e-5, method=method)
    a, b = cuda.tensor(s, device="cuda"), cuda.tensor(s, device="cuda")
    stream = cuda.cuda.Stream()
    stream.wait_stream(cuda.cuda.current_stream())
    with BIASolver(stream=stream) as solver:
        solver.step(a, cfg, stats=False)
    ptrs = [ctypes.c_void_p(b.data_ptr() + 8 * n * k) for k in range(6)]
    assert capi.lib().bia_step_noalloc(ctypes.byref(cfg), n, *ptrs, None, None,
                                       ctypes.c_void_p(stream.cuda_stream)) == capi.BIA_OK
    stream.synchronize()
    assert cuda.equal(a, b)


CHILD = """
import ctypes, sys
import numpy as np
from bia_3d_gpu_b200 import METHOD_ALG, METHOD_RKF, METHOD_UNIVERSAL, capi, default_config, initial

cu = ctypes.CDLL("libcuda.so.1")


def ok(r):
    assert r == 0, r


dev, ctx = ctypes.c_int(), ctypes.c_void_p()
ok(cu.cuInit(0))
ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
n = 257
s, eps = initial.plummer(n, seed=63)


def retain():
    ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), dev))
    ok(cu.cuCtxSetCurrent(ctx))


def steps(method, make_context):
    cfg = default_config(eps_th=eps, dt=1e-5, method=method)
    ptr = ctypes.c_uint64()
    ok(cu.cuMemAlloc_v2(ctypes.byref(ptr), s.nbytes))
    ok(cu.cuMemcpyHtoD_v2(ptr, s.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(s.nbytes)))
    rows = [ctypes.c_void_p(ptr.value + 8 * n * k) for k in range(6)]
    if make_context:
        c = ctypes.c_void_p()
        capi.check(capi.lib().bia_context_create(ctypes.byref(c), 0, None), "bia_context_create")
        capi.check(capi.lib().bia_step(c, ctypes.byref(cfg), n, *rows, None, None, None), "bia_step")
        capi.lib().bia_context_destroy(c)
    else:
        capi.check(capi.lib().bia_step_noalloc(ctypes.byref(cfg), n, *rows, None, None, None), "bia_step_noalloc")
    out = np.empty_like(s)
    ok(cu.cuCtxSynchronize())
    ok(cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), ptr, ctypes.c_size_t(s.nbytes)))
    return out


def every(order):
    return {(m, c): steps(m, c) for c in order for m in (METHOD_ALG, METHOD_RKF, METHOD_UNIVERSAL)}


retain()
before = every((False, True))
for order in ((False, True), (True, False)):
    ok(cu.cuDevicePrimaryCtxRelease_v2(dev))
    ok(cu.cuDevicePrimaryCtxReset_v2(dev))
    retain()
    after = every(order)
    for k in before:
        assert np.array_equal(before[k], after[k]), k
print("same steps after a reset")
"""


def test_steps_after_a_context_reset(cuda):
    p = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "same steps after a reset" in p.stdout, p.stdout + p.stderr
