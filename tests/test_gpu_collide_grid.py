"""The collision update's grid form against the oracle's ordered reflections,
bit for bit: its smallest size and one below, bodies on both sides of zero and
on cell edges, rows of cells that leave a block of buckets, more contacts than
a target can list, and a body that no cell holds (the other forms then)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def layout(kind, n):
    rng = np.random.default_rng(n)
    if kind == "line":  # one row of cells, the longest run of buckets
        pos = np.zeros((n, 3))
        pos[:, 0] = rng.uniform(-0.004 * n, 0.004 * n, n)
    elif kind == "edges":  # multiples of the cell edge and of the contact distance
        pos = rng.integers(-12, 12, (n, 3)) * np.where(rng.random((n, 1)) < 0.5, 0.031875, 0.03)
    else:
        pos = rng.uniform(-1, 1, (n, 3))
        if kind == "clump":  # a dense core: its targets overflow their lists
            pos[: n // 8] *= 0.03
        if kind == "far":
            pos[n // 2, 1] = 3.0e4
    return pos.astype(np.float32)


@pytest.mark.parametrize("kind,n", [("uniform", 5119), ("uniform", 5120), ("line", 5121), ("edges", 5999),
                                    ("uniform", 33333), ("clump", 20001), ("far", 6001)])
@pytest.mark.parametrize("algo", [0, 2])
def test_grid_form_bit_exact(gpu, oracle, kind, n, algo):
    nb = gpu
    pos = layout(kind, n)
    if algo == 0 and kind in ("line", "edges"):
        pytest.skip("coincident bodies have no tree")
    vel = (0.1 * np.random.default_rng(n + 1).normal(size=(n, 3))).astype(np.float32)
    sim = nb.Simulation(num_of_bodies=n, algo_config=algo, collision=1, gravitational_constant=0.0)
    sim.set_state(pos, np.full(n, 1.0 / n, np.float32), vel)
    sim.step(0.0, 1)  # no gravity, no drift: the collision update alone
    want = oracle.collision(pos, vel)
    assert np.any(want != vel)
    assert np.array_equal(sim.get_state()[1], want)
