"""Bodies without mass (tracers) that have a cell to themselves: its centre of
mass is not a number, so no distance accepts it and the walk opens it.  Cells so
small that the opening distance is the softening alone (a cluster of tracers a
millionth across), and softenings above one with the reference's opening rule,
where the squared softening exceeds the rule's."""
import numpy as np
import pytest


def bodies(kind, n=3000):
    rng = np.random.default_rng(n + len(kind))
    pos = rng.normal(size=(n, 3)).astype(np.float32)
    mass = (rng.random(n) + 0.5).astype(np.float32)
    if kind == "cluster":
        few = slice(100, 140)
        pos[few] = np.float32(0.25) + np.float32(2.0 ** -25) * rng.integers(0, 32, (40, 3)).astype(np.float32)
        mass[few] = 0.0
    else:
        mass[: n // 2] = 0.0
    return pos, mass / mass.sum()


CASES = [("cluster", 0.05, 0), ("scattered", 2.0, 1), ("scattered", 0.01, 0)]


def expected(oracle, kind, eps, crit, quad, comp, nodes=None):
    pos, mass = bodies(kind)
    rule = oracle.CRIT_REFERENCE if crit else oracle.CRIT_STANDARD
    acc = oracle.bh_step_forces(pos, mass, 0.6, eps, 1.0, criterion=rule, nodes=nodes, quadrupole=bool(quad),
                                compensated=bool(comp))[0]
    assert np.isfinite(acc).all()
    return pos, mass, acc.astype(np.float64)


@pytest.mark.parametrize("kind,eps,crit", CASES)
def test_oracle_opens_massless_cells(oracle, kind, eps, crit):
    expected(oracle, kind, eps, crit, 0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,eps,crit", CASES)
@pytest.mark.parametrize("quad,comp", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_massless_cells(gpu, oracle, kind, eps, crit, quad, comp):
    nb = gpu
    pos, mass = bodies(kind)
    n = len(mass)
    cfg = nb.default_config(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.6, epsilon=eps,
                            gravitational_constant=1.0, multipole=quad, precision=comp, theta_semantics=crit)
    with nb.Simulation(cfg) as s:
        s.set_state(pos, mass)
        s.step(0.0, 1)
        got = s.get_state()[2]
        _, _, want = expected(oracle, kind, eps, crit, quad, comp, int(s.stage_debug(nb.DEBUG_TREE_INFO)[1]))
    # 2e-5 of the typical |a|: sums of at most n FP32 terms, each within 1e-6 of
    # the oracle's (MUFU rsqrt, another order), on the same interactions
    scale = np.sqrt(np.mean(np.sum(want ** 2, axis=1)))
    assert np.max(np.linalg.norm(got - want, axis=1)) < 2e-5 * scale
    with nb.Batch([cfg]) as b:
        b.set_state(0, pos, mass)
        b.step(0.0, 1)
        np.testing.assert_array_equal(b.get_state(0)[2], got)
