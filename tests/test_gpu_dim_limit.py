"""Which kernel bia_dim_integrate takes on both sides of the resident kernel's limit, 224 particles (7 a lane, 32
lanes) a CTA and a CTA per SM, without the environment's cap on the blocks: one particle above the limit the run is
bitwise that of the kernel with its state in global memory, at the limit it is not, and agrees to 1e-13."""
import numpy as np
import pytest

from bia_3d_gpu_b200 import BIASolver, initial
from conftest import max_rel_err, rel_err

pytestmark = pytest.mark.gpu


def _run(cuda, s, eps, xe):
    t = cuda.tensor(s, device="cuda")
    with BIASolver() as solver:
        st = solver.dim_integrate(t, eps, 0.0, xe)
        solver.stream.synchronize()
    return t.cpu().numpy(), st


@pytest.mark.parametrize("above", [0, 1])
def test_limit_of_the_resident_kernel(cuda, above, monkeypatch):
    monkeypatch.delenv("BIA_DIM_COOP_BLOCKS", raising=False)
    n = 224 * cuda.cuda.get_device_properties(0).multi_processor_count + above
    s, eps = initial.plummer(n, seed=12)
    got, st = _run(cuda, s, eps / 2, 1e-6)
    monkeypatch.setenv("BIA_DIM_COOP_BLOCKS", "1024")  # as many as that kernel has: no cap, and not the resident one
    ref, rst = _run(cuda, s, eps / 2, 1e-6)
    assert st["ier"] == 0 and st["accepted"] == rst["accepted"] and st["nde"] == rst["nde"]
    assert np.array_equal(got, ref) == bool(above)
    for part in (slice(0, 3), slice(3, 6)):
        assert rel_err(got[part], ref[part]) <= 1e-13 and max_rel_err(got[part], ref[part]) <= 1e-13
