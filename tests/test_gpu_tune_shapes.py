"""The autotuner chooses what the timed steps show: the two parameters of
insertions (top levels, bodies per block) keep their defaults in a batch whose
trees come from sorted paths, and are chosen where a tree inserts; the state and
the results are the same either way."""
import numpy as np
import pytest

from test_gpu_batch import cfg
from test_gpu_build import bodies

pytestmark = pytest.mark.gpu


def tuned(nb, kind, sizes):
    with nb.Batch([cfg(nb, n, True, 3) for n in sizes]) as b:
        untuned = None
        for tune in (False, True):
            for k, n in enumerate(sizes):
                b.set_state(k, *bodies(kind, n))
            if tune:
                b.autotune()
            b.step(1e-4, 2)
            got = [b.get_state(k)[:2] for k in range(len(sizes))]
            if untuned is None:
                untuned = got
            for g, w in zip(got, untuned):
                np.testing.assert_array_equal(g[0], w[0])
                np.testing.assert_array_equal(g[1], w[1])
        return b.tree_shape()


def test_batch_without_insertions(gpu):
    for n in (1500, 3000, 6007, 9001, 20000, 30000):
        shape = tuned(gpu, "ball", [n] * 6)
        assert (shape["build_chunk"], shape["top_levels"]) == (0, 4), n


def test_batch_with_insertions(gpu):
    shape = tuned(gpu, "outlier", [20000] * 4)
    assert shape["build_chunk"] in (0, 1024, 2048, 4096) and shape["top_levels"] in (0, 2, 3, 4)
