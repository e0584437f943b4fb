"""Trees of a batch from sorted octant paths, and the insertions that some of
its systems take: sizes around a tile of 256 and an entry of 1,024 bodies and
around the changes of the region levels, beside crowded regions, points that
21 levels do not part and the reference's tree semantics.  Every system steps
as a standalone handle does, bit for bit."""
import numpy as np
import pytest

from test_gpu_batch import cfg, standalone
from test_gpu_build import bodies

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 7, 127, 128, 255, 256, 257, 1023, 1024, 1025, 2049, 8191, 8192, 65535, 65537)
SPECIAL = [("clumps", 30001), ("outlier", 5000), ("outlier", 60001), ("close", 700), ("close", 20000), ("plane", 10007)]


def compare(nb, specs, steps, method=3, quad=0):
    cfgs, states = [], []
    for kind, n, ref in specs:
        c = cfg(nb, n, True, method=method, quad=quad)
        if ref:
            c.tree_semantics = nb.TREE_REFERENCE
        pos, mass = bodies(kind, n)
        cfgs.append(c)
        states.append((pos, mass, np.zeros_like(pos)))
    with nb.Batch(cfgs) as b:
        for k, (p, m, v) in enumerate(states):
            b.set_state(k, p, m, v)
        b.step(1e-3, steps, check=False)
        for k, (p, m, v) in enumerate(states):
            with nb.Simulation(cfgs[k]) as s:
                s.set_state(p, m, v)
                assert s.step(1e-3, steps, check=False) == b.system_status(k), specs[k]
                want = s.get_state()
            for g, w in zip(b.get_state(k)[:2], want[:2]):
                np.testing.assert_array_equal(g, w, err_msg=str(specs[k]))


@pytest.mark.parametrize("quad", [0, 1])
def test_sizes(gpu, quad):
    compare(gpu, [("ball", n, False) for n in SIZES], 3, quad=quad)


@pytest.mark.parametrize("quad", [0, 1])
def test_systems_that_insert(gpu, quad):
    plain = [("ball", n, False) for n in (300, 4096, 40000)]
    refs = [("ball", n, True) for n in (1, 500, 7000)]
    compare(gpu, plain + [(kind, n, False) for kind, n in SPECIAL] + refs, 3, quad=quad)


def test_only_reference_trees(gpu):
    compare(gpu, [("ball", n, True) for n in (2, 3000, 20000)], 2, method=2)


def test_reference_trees_around_the_switch_to_insertions(gpu):
    compare(gpu, [("ball", n, True) for n in (131072, 131073)] + [("ball", 5000, False), ("outlier", 6000, False)], 2)


def test_a_tree_without_cells_left(gpu):
    """One system overflows its cells and keeps its state; the others step on."""
    nb = gpu
    sizes = (5000, 3000, 9000)
    cfgs = [cfg(nb, n, True, cap=64 if k == 1 else 0) for k, n in enumerate(sizes)]
    states = [bodies("ball", n) for n in sizes]
    with nb.Batch(cfgs) as b:
        for k, (p, m) in enumerate(states):
            b.set_state(k, p, m)
        with pytest.raises(Exception):
            b.step(1e-3, 2)
        np.testing.assert_array_equal(b.get_state(1)[0], states[1][0])
        for k in (0, 2):
            want = standalone(nb, cfgs[k], *states[k], None, 1e-3, 2)
            np.testing.assert_array_equal(b.get_state(k)[0], want[0])
