"""Steps of large trees with the reference's semantics, whose stages are kernels
of their own, from several threads at once: none of their blocks waits for
another, so they finish beside one another, each with what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n):
    rng = np.random.default_rng(n)
    return rng.normal(size=(n, 3)).astype(np.float32), np.full(n, 1.0 / n, np.float32)


def run_together(work):
    """Every function of `work` in a thread of its own, from a common start; their
    results in order."""
    out, start = [None] * len(work), threading.Barrier(len(work))

    def run(k):
        start.wait()
        out[k] = work[k]()

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return out


def test_large_reference_trees(gpu):
    nb = gpu
    sizes = (131073, 150001, 131073, 200003)
    sims = []
    for n in sizes:
        s = nb.Simulation(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.7, epsilon=0.01,
                          gravitational_constant=1.0, tree_semantics=nb.TREE_REFERENCE)
        s.set_state(*system(n))
        sims.append(s)
    alone = []
    for s, n in zip(sims, sizes):
        assert s.step(1e-4, 6, check=False) == 0
        alone.append(s.get_state()[:2])
        s.set_state(*system(n))
    together = run_together([lambda s=s: (s.step(1e-4, 6, check=False), s.get_state()[:2]) for s in sims])
    for (status, got), want in zip(together, alone):
        assert status == 0
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    for s in sims:
        s.close()
