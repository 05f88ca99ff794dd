"""DIM from several host threads, each with its own context (bia_dim_integrate) or its thread's own buffers
(rkf_c_): a larger system among smaller ones that run the same form of the resident kernel with less
shared memory (one particle a lane: 59 and 53 KB on 148 SMs).  Every call succeeds and gives the single-threaded bits.
The threads share a stream: what a call sets for its launch is set on the host, and that is tested."""
import threading

import numpy as np
import pytest

from bia_3d_gpu_b200 import BIASolver, initial, rkf_c

pytestmark = pytest.mark.gpu

SIZES = [1000] + 7 * [200]
CALLS = 400


# Each yields a call that integrates the system once: its state and its steps or derivatives.
def _dim(cuda, stream, s, eps, xe):
    with BIASolver(stream=stream) as solver:
        def call():
            t = cuda.tensor(s, device="cuda")
            st = solver.dim_integrate(t, eps, 0.0, xe)
            return t.cpu().numpy(), st["accepted"]
        yield call


def _rkf_c(cuda, stream, s, eps, xe):
    y0 = np.ascontiguousarray(s.T).reshape(-1)

    def call():
        out = rkf_c(y0.size, eps, 0.0, xe, y0.copy(), 1, 0.0, 1e-16)
        return out["YHN"], out["NDE"]
    yield call


@pytest.mark.parametrize("entry", [_dim, _rkf_c])
def test_threads_of_different_sizes(cuda, entry):
    xe = 1e-7
    stream = cuda.cuda.Stream()
    systems = {n: initial.plummer(n, seed=n) for n in set(SIZES)}
    want = {n: [call() for call in entry(cuda, stream, s, eps / 2, xe)][0] for n, (s, eps) in systems.items()}
    wrong = []
    done = threading.Event()

    def work(n, calls):
        s, eps = systems[n]
        for call in entry(cuda, stream, s, eps / 2, xe):
            while calls != 0 and not done.is_set():
                calls -= 1
                try:
                    got = call()
                except Exception as e:  # a refused call
                    wrong.append((n, repr(e)))
                    continue
                if not (np.array_equal(got[0], want[n][0]) and got[1] == want[n][1]):
                    wrong.append((n, "other bits"))

    # the first makes its calls, the others go on until it has
    threads = [threading.Thread(target=work, args=(n, CALLS if k == 0 else -1)) for k, n in enumerate(SIZES)]
    for t in threads:
        t.start()
    threads[0].join()
    done.set()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:3])
