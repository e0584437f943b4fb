"""Walks whose stacks grow long (the reference's opening rule opens every cell
within sqrt(eps), so a dense centre is opened all the way down): against the
oracle, alone and in a batch, and in a time that the number of its rounds
explains."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cusp(n):
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    pos = d / np.linalg.norm(d, axis=1)[:, None] * 10.0 ** rng.uniform(-4, 1, (n, 1))
    mass = (rng.random(n) + 0.5).astype(np.float32)
    return pos.astype(np.float32), mass / mass.sum()


def config(nb, n, quad=0, comp=0, eps=0.001, **kw):
    return nb.default_config(num_of_bodies=n, theta=0.5, epsilon=eps, gravitational_constant=1.0, multipole=quad,
                             precision=comp, theta_semantics=nb.THETA_REFERENCE, **kw)


@pytest.mark.parametrize("n", [700, 6869])
@pytest.mark.parametrize("quad,comp", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_cusp_against_oracle(gpu, oracle, n, quad, comp):
    nb = gpu
    pos, mass = cusp(n)
    eps = 0.01  # the closest pairs do not decide the comparison
    cfg = config(nb, n, quad, comp, eps, algo_config=nb.BARNES_HUT)
    with nb.Simulation(cfg) as s:
        s.set_state(pos, mass)
        s.step(0.0, 1)
        got = s.get_state()[2]
        nodes = int(s.stage_debug(nb.DEBUG_TREE_INFO)[1])
        want, tree, _ = oracle.bh_step_forces(pos, mass, 0.5, eps, 1.0, criterion=oracle.CRIT_REFERENCE, nodes=nodes,
                                              quadrupole=bool(quad), compensated=bool(comp))
        assert s.work_counters()[1] > 20 * ((n + 31) // 32)  # dozens of cells opened a group
    scale = np.sqrt(np.mean(np.sum(want.astype(np.float64) ** 2, axis=1)))
    # as the other walks: 2e-5 of the typical |a|
    assert np.max(np.linalg.norm(got.astype(np.float64) - want, axis=1)) < 2e-5 * scale
    with nb.Batch([cfg]) as b:
        b.set_state(0, pos, mass)
        b.step(0.0, 1)
        np.testing.assert_array_equal(b.get_state(0)[2], got)


def test_long_stacks_are_popped_in_batches(gpu):
    """Against the direct sum of the same bodies, whose time follows the clock the
    same way: seven times its 0.17 ms; with single pops from 128 entries on 24 times."""
    nb = gpu
    n = 20000
    ms = []
    for cfg in (config(nb, n, 1, 0, 0.01, algo_config=nb.BARNES_HUT, tree_semantics=nb.TREE_REFERENCE),
                config(nb, n, 0, 0, 0.01, algo_config=nb.BRUTE_FORCE_LOCAL)):
        with nb.Simulation(cfg) as s:
            s.set_state(*cusp(n))
            s.step(0.0, 2)
            s.set_profiling(True)
            took = []
            for _ in range(9):
                s.step(0.0, 1)
                t = s.timings()
                took.append(t["force"] + t["direct"])
            ms.append(min(took))
    assert ms[0] < 14.0 * ms[1]


@pytest.mark.parametrize("quad", [0, 1])
def test_deep_tree_and_wide_stack(gpu, oracle, quad):
    """Pairs that part at every level down to the deepest the walk takes, between
    bodies whose cells are all opened: the least room for batches."""
    nb = gpu
    rng = np.random.default_rng(5)
    k = np.arange(118) // 2
    deep = np.ldexp(1.0, -k)[:, None] * (1.0 + 0.25 * (np.arange(118) % 2)[:, None]) * np.array([[1.0, 0.75, 0.5]])
    pos = np.concatenate([deep, 0.02 * rng.normal(size=(3000, 3))]).astype(np.float32)
    mass = np.full(len(pos), 1.0 / len(pos), np.float32)
    cfg = config(nb, len(pos), quad, 0, 0.01, algo_config=nb.BARNES_HUT)
    with nb.Simulation(cfg) as s:
        s.set_state(pos, mass)
        s.step(0.0, 1)
        info = s.stage_debug(nb.DEBUG_TREE_INFO)
        got = s.get_state()[2].astype(np.float64)
    assert int(info[3]) > 55
    want = oracle.bh_step_forces(pos, mass, 0.5, 0.01, 1.0, criterion=oracle.CRIT_REFERENCE, nodes=int(info[1]),
                                 quadrupole=bool(quad))[0].astype(np.float64)
    scale = np.sqrt(np.mean(np.sum(want ** 2, axis=1)))
    assert np.max(np.linalg.norm(got - want, axis=1)) < 2e-5 * scale
