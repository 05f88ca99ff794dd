"""bia_invariance at the edges of its units (two 32-particle block rows of a block column) and of its grid, with
and without charges, against the quad-precision invariants of the oracle: a few hundred roundings of
positive terms (1e-13; the pair sum of mixed charges on the scale of its magnitudes), the same bits on a
second call, and coincident particles (an infinite pair sum, as 1/r gives it)."""
import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import BIASolver, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 129, 161, 700, 1333, 3001])
@pytest.mark.parametrize("charged", [False, True])
def test_invariants_match_quad_oracle(cuda, n, charged):
    if charged and n > 1:
        s, eps, q = initial.coulomb_cube(n, seed=n, dmin=1e-3)
    else:
        s, eps = initial.plummer(n, seed=n)
        q = None
    ref = oracle.invariance(s, eps, q=q, quad=True) if q is not None else oracle.invariance(s, eps, quad=True)
    t = cuda.tensor(s, device="cuda")
    qt = None if q is None else cuda.tensor(q, device="cuda")
    with BIASolver() as solver:
        a = solver.invariance(t, eps, q=qt)
        b = solver.invariance(t, eps, q=qt)
    assert a == b
    d = np.sqrt(((s[:3, :, None] - s[:3, None, :]) ** 2).sum(0))
    size = {"KE": (s[3:] ** 2).sum(), "PE": abs(eps) * (1.0 / d[np.triu_indices(n, 1)]).sum()}
    for k in ("Lx", "Ly", "Lz"):
        size[k] = (np.abs(s[:3]).max(0) * np.abs(s[3:]).max(0)).sum()
    for k, row in zip(("Ua", "Va", "Wa", "Xa", "Ya", "Za"), (3, 4, 5, 0, 1, 2)):
        size[k] = np.abs(s[row]).sum()
    for k, v in size.items():
        assert abs(a[k] - ref[k]) <= 1e-13 * max(v, 1e-300), k


def test_coincident_particles_give_an_infinite_sum(cuda):
    s, eps = initial.plummer(40, seed=2)
    s[:3, 7] = s[:3, 35]
    with BIASolver() as solver:
        out = solver.invariance(cuda.tensor(s, device="cuda"), 2.0)
    assert out["PE"] == np.inf and np.isfinite(out["KE"])
