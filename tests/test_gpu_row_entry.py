"""The per-particle drop-in row at the edges of its warps, against the oracle's rows: the last
particle (no pair), one pair, 31 to 33 and 64 + 1 pairs, buffers reused by shorter and by longer
calls, input and output in one array, and calls from threads that end."""
import threading

import numpy as np
import pytest

import oracle
from bia_3d_gpu_b200 import find_dxyuv_kernel, initial

pytestmark = pytest.mark.gpu

DT = 1e-4


def row(method, s, eps, i, alias=False):
    n = s.shape[1]
    acc = np.zeros((6, n))
    rel = np.ascontiguousarray((s[:, i : i + 1] - s).T).reshape(-1)
    out = rel if alias else np.full(6 * n, np.nan)
    assert find_dxyuv_kernel(method, n, i + 1, eps, DT, 18, *acc, rel, out) == 0
    return acc, out.reshape(n, 6).T


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 32, 33, 34, 66, 40])
def test_row_edges(cuda, method, n):
    s, eps = initial.plummer(70, seed=51)
    s = np.ascontiguousarray(s[:, :n])
    for i in sorted({0, n // 2, n - 1}):
        acc, h = row(method, s, eps, i)
        assert np.all(h[:, : i + 1] == 0)
        assert np.array_equal(acc[:, i + 1 :], -h[:, i + 1 :])
        # a sum of m terms in any order: m units of rounding of the sum of magnitudes
        assert np.all(np.abs(acc[:, i] - h.sum(1)) <= n * 2.3e-16 * np.abs(h).sum(1))
        # the oracle ends a solve when its angle moves by less than 1e-12 of itself; each of the
        # m pairs may be off by that much of its relative state
        want, _, _ = oracle.bia_rows(s, eps, DT, [i], method=method)
        scale = np.abs(s[:, i : i + 1] - s).reshape(2, 3, n).max((1, 2)).repeat(3)[:, None]
        assert np.all(np.abs(acc - want) <= 1e-12 * n * scale)
        again, h2 = row(method, s, eps, i, alias=True)
        assert np.array_equal(h, h2) and np.array_equal(acc, again)


def test_row_threads_reuse_buffers(cuda):
    s, eps = initial.plummer(70, seed=51)
    want = row(1, s, eps, 3)[1]
    got = []
    for _ in range(3):
        ts = [threading.Thread(target=lambda: got.append(row(1, s, eps, 3)[1])) for _ in range(3)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    assert len(got) == 9 and all(np.array_equal(g, want) for g in got)
