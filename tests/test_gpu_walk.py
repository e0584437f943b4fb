"""The force walk where its lists and entries are at their edges: lists of
every remainder of the tile size, groups whose bounding box decides little
(two far clusters in one warp), and cells more than 32 levels deep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(layout, n):
    rng = np.random.default_rng(n)
    mass = (rng.random(n) + 0.5).astype(np.float32)
    mass /= mass.sum()
    if layout == "pile":  # pairs of bodies that part one level deeper each: 2^-k
        k = np.arange(n) // 2
        pos = np.ldexp(1.0, -k)[:, None] * (1.0 + 0.25 * (np.arange(n) % 2)[:, None]) * np.array([[1.0, 0.75, 0.5]])
    elif layout == "two":  # two small clusters far apart, interleaved in one warp group
        pos = 0.05 * rng.normal(size=(n, 3)) + np.where(np.arange(n) % 2, 3.0, -3.0)[:, None]
    else:
        pos = rng.normal(size=(n, 3))
    return pos.astype(np.float32), mass


# 2e-5 of the typical |a|: sums of at most n FP32 terms, each within 1e-6 of
# the oracle's (MUFU rsqrt, another order), on the same interactions
@pytest.mark.parametrize("layout,n", [("pile", 90), ("two", 40), ("two", 700), ("normal", 9), ("normal", 15),
                                      ("normal", 47), ("normal", 1500)])
@pytest.mark.parametrize("quad,comp", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_walk_edges(gpu, oracle, layout, n, quad, comp):
    nb = gpu
    pos, mass = bodies(layout, n)
    sim = nb.Simulation(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.6, epsilon=0.01,
                        gravitational_constant=1.0, multipole=quad, precision=comp)
    sim.set_state(pos, mass)
    sim.step(0.0, 1)
    info = sim.stage_debug(nb.DEBUG_TREE_INFO)
    if layout == "pile":
        assert int(info[3]) > 32
    acc_o, _, _ = oracle.bh_step_forces(pos, mass, 0.6, 0.01, 1.0, nodes=int(info[1]), quadrupole=bool(quad),
                                        compensated=bool(comp))
    acc = sim.get_state()[2].astype(np.float64)
    scale = np.sqrt(np.mean(np.sum(acc_o.astype(np.float64) ** 2, axis=1)))
    assert np.max(np.linalg.norm(acc - acc_o, axis=1)) < 2e-5 * scale


@pytest.mark.parametrize("quad,comp", [(0, 0), (0, 1), (1, 1)])
def test_walk_of_many_groups(gpu, quad, comp):
    """The walk with more warps per SM, which systems take whose groups fill the
    GPU twice over (152 SMs: 4,864 groups): bit for bit the batched walk, which
    has one form."""
    nb = gpu
    sizes = (155616, 155617, 200000)
    cfgs = [nb.default_config(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.8, epsilon=0.01,
                              gravitational_constant=1.0, multipole=quad, precision=comp) for n in sizes]
    states = [bodies("normal", n) for n in sizes]
    with nb.Batch(cfgs) as b:
        for k, (pos, mass) in enumerate(states):
            b.set_state(k, pos, mass)
        b.step(1e-3, 1)
        for k, (pos, mass) in enumerate(states):
            with nb.Simulation(cfgs[k]) as sim:
                sim.set_state(pos, mass)
                sim.step(1e-3, 1)
                for one, batched in zip(sim.get_state(), b.get_state(k)):
                    np.testing.assert_array_equal(one, batched)
