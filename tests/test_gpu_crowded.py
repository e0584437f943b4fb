"""Crowded regions of the build from sorted paths (most bodies in few of them, as
when one body is far out): around the number of bodies in one region from which
the step takes the insertions, the tree, its sort and the step are those of the
insertions, bit for bit; and ranking a crowd never costs what the insertions do
not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crowd(n, many):
    """`many` of n bodies in one region of the first levels, the others spread: odd
    multiples of 2^-23, so that no body lies on a plane between cells of the first
    20 levels (where the reference's semantics take it to one side and its box to
    the other, and the tree depends on the order of the insertions)."""
    rng = np.random.default_rng(n + many)
    pos = rng.uniform(-1, 1, (n, 3))
    at = rng.permutation(n)[:many]
    pos[at] = np.array([0.70, 0.45, 0.58]) + 1e-2 * rng.uniform(-1, 1, (many, 3))
    pos = (2.0 * np.floor(pos * 2.0 ** 22) + 1.0) * 2.0 ** -23
    pos[0], pos[1] = (-1, -1, -1), (1, 1, 1)
    return pos.astype(np.float32)


def limit(n, ref):  # build_device.cuh, crowd_limit
    return n if not ref and n <= 4096 else 2048 + n // 64


def handle(nb, n, pos, ref=0, theta=0.7):
    s = nb.Simulation(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=theta, epsilon=0.01, gravitational_constant=1.0,
                      tree_semantics=ref)
    s.set_state(pos, np.full(n, 1.0 / n, np.float32))
    return s


@pytest.mark.parametrize("n", [2600, 4096, 4097, 9001, 60001, 262145])
@pytest.mark.parametrize("more", [-1, 0, 1, 2, 700])
@pytest.mark.parametrize("ref", [0, 1])
def test_around_the_limit(gpu, n, more, ref):
    nb = gpu
    if ref and n > 131072:
        pytest.skip("such a tree has kernels of its own")
    pos = crowd(n, min(limit(n, ref) + more, n - 2))
    got = []
    for insert in (False, True):
        with handle(nb, n, pos, ref) as s:
            if insert:
                s.set_spin_cap(1 << 22)
            status = [s.step(0.0, 1, check=False) for _ in range(2)]
            info = s.stage_debug(nb.DEBUG_TREE_INFO)
            got.append((status, int(info[2]), int(info[3]), s.stage_debug(nb.DEBUG_SORTED), *s.get_state()))
    assert got[0][:3] == got[1][:3] and got[0][0] == [0, 0]
    for a, b in zip(got[0][3:], got[1][3:]):
        np.testing.assert_array_equal(a, b)


def test_batched_crowds(gpu):
    nb = gpu
    sizes = [(n, limit(n, 0) + more) for n in (4097, 9001, 60001) for more in (0, 1, 500)]
    cfgs = [nb.default_config(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.7, epsilon=0.01,
                              gravitational_constant=1.0) for n, _ in sizes]
    with nb.Batch(cfgs) as b:
        for k, (n, many) in enumerate(sizes):
            b.set_state(k, crowd(n, many), np.full(n, 1.0 / n, np.float32))
        b.step(1e-4, 3)
        for k, (n, many) in enumerate(sizes):
            with handle(nb, n, crowd(n, many)) as s:
                s.step(1e-4, 3)
                for one, batched in zip(s.get_state(), b.get_state(k)):
                    np.testing.assert_array_equal(one, batched)


def test_a_crowd_is_not_ranked_for_long(gpu):
    """20,000 normal bodies and one 100 units out, which leaves nearly all of them
    in few regions, against one 200 units out, whose step inserts at once."""
    nb = gpu
    n, ms = 20000, []
    for far in (200.0, 100.0):
        pos = np.random.default_rng(n).normal(size=(n, 3)).astype(np.float32)
        pos[0] = (far, -0.75 * far, 0.5 * far)
        with handle(nb, n, pos) as s:
            s.step(0.0, 1)
            s.set_profiling(True)
            took = []
            for _ in range(9):
                s.step(0.0, 1)
                t = s.timings()
                took.append(sum(t[k] for k in ("bbox", "build", "summarize", "sort")))
            ms.append(min(took))
    assert ms[1] < 1.6 * ms[0]  # 0.17 ms both; ranked 0.41
