"""Steps whose trees take the insertions, of several handles and batches at once
from threads of their own: their kernels hold the GPU beside one another, each
finishes, and each gives what it gives alone."""
import threading

import numpy as np
import pytest

from test_gpu_batch import cfg
from test_gpu_build import bodies

pytestmark = pytest.mark.gpu


def test_insertions_side_by_side(gpu):
    nb = gpu
    n, calls = 60001, 3
    pos, mass = bodies("outlier", n)

    def run_sim(s, out, k):
        s.set_state(pos, mass)
        out[k] = [s.step(1e-4, 2, check=False) for _ in range(calls)], s.get_state()[:2]

    def run_batch(b, out, k):
        for j in range(4):
            b.set_state(j, pos, mass)
        out[k] = [b.step(1e-4, 2, check=False) for _ in range(calls)], b.get_state(3)[:2]

    # created one after another (creation synchronises the device, which another
    # thread's graph capture does not allow), then stepped together
    work = [(run_batch, nb.Batch([cfg(nb, n, True, method=3)] * 4)) if k in (1, 3) else
            (run_sim, nb.Simulation(cfg(nb, n, True, method=3))) for k in range(6)]
    alone, out = {}, {}
    run_sim(work[0][1], alone, 0)
    assert alone[0][0] == [0] * calls
    threads = [threading.Thread(target=run, args=(handle, out, k)) for k, (run, handle) in enumerate(work)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, (_, handle) in enumerate(work):
        assert out[k][0] == alone[0][0]
        for got, want in zip(out[k][1], alone[0][1]):
            np.testing.assert_array_equal(got, want)
        handle.close()
