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
    n, steps = 60001, 6
    pos, mass = bodies("outlier", n)

    def sim_run(out, k):
        with nb.Simulation(cfg(nb, n, True, method=3)) as s:
            s.set_state(pos, mass)
            status = [s.step(1e-4, 2, check=False) for _ in range(steps // 2)]
            out[k] = (status, s.get_state()[:2])

    def batch_run(out, k):
        with nb.Batch([cfg(nb, n, True, method=3)] * 4) as b:
            for j in range(4):
                b.set_state(j, pos, mass)
            status = [b.step(1e-4, 2, check=False) for _ in range(steps // 2)]
            out[k] = (status, b.get_state(3)[:2])

    alone = {}
    sim_run(alone, 0)
    assert alone[0][0] == [0] * (steps // 2)
    out = {}
    threads = [threading.Thread(target=run, args=(out, k)) for k, run in
               enumerate([sim_run, batch_run, sim_run, batch_run, sim_run, sim_run])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(threads)):
        assert out[k][0] == alone[0][0]
        for got, want in zip(out[k][1], alone[0][1]):
            np.testing.assert_array_equal(got, want)
