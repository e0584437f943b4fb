"""Handles and batches of several threads at once, each of which gives what it
gives alone: steps of large trees with the reference's semantics, whose stages
are kernels of their own and none of whose blocks waits for another, and handles
created and closed while other threads capture the graphs of their first steps."""
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


def test_created_and_closed_side_by_side(gpu):
    nb = gpu
    n, rounds = 6007, 12
    pos, mass = system(n)
    kind = dict(theta=0.7, epsilon=0.01, gravitational_constant=1.0)
    tree = nb.default_config(num_of_bodies=n, algo_config=nb.BARNES_HUT, **kind)
    direct = nb.default_config(num_of_bodies=n, algo_config=nb.BRUTE_FORCE_LOCAL, **kind)

    def handle(cfg):
        got = []
        for _ in range(rounds):
            with nb.Simulation(cfg) as s:
                s.set_state(pos, mass)
                got.append((s.step(1e-3, 2, check=False), s.get_state()[:2]))
        return got

    def batch(cfg):
        got = []
        for _ in range(rounds):
            with nb.Batch([cfg, cfg]) as b:
                b.set_state(0, pos, mass)
                b.set_state(1, pos, mass)
                got.append((b.step(1e-3, 2, check=False), b.get_state(1)[:2]))
        return got

    def server(cfg):
        got = []
        for _ in range(rounds):
            with nb.Server(max_jobs=4, snapshot_every=0) as v:
                ids = [v.submit(cfg, 2, 1e-3, pos, mass) for _ in range(3)]
                got.append((v.wait(), v.result(ids[-1], n)))
        return got

    work = [lambda: handle(tree), lambda: batch(tree), lambda: handle(direct), lambda: batch(direct),
            lambda: server(tree), lambda: batch(tree), lambda: handle(tree), lambda: batch(tree)]
    alone = {k: work[k]()[0] for k in range(5)}
    alone |= {5: alone[1], 6: alone[0], 7: alone[1]}
    for k, results in enumerate(run_together(work)):
        assert results is not None, k
        for status, got in results:
            assert status == 0, k
            for g, w in zip(got, alone[k][1]):
                np.testing.assert_array_equal(g, w)
