"""Systems whose targets the collision grid cannot serve (a body that no cell
holds, a system or a core so dense that targets have more contacts than their
lists hold) take the all-pairs forms behind it: bit for bit the oracle's ordered
reflections, in little more time than a system that is just too small for the
grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def layout(kind, n):
    rng = np.random.default_rng(3)
    d = rng.normal(size=(n, 3))
    pos = d / np.linalg.norm(d, axis=1)[:, None] * rng.random((n, 1)) ** (1 / 3)  # unit ball
    if kind == "far":
        pos[n // 2, 1] = 3.0e4
    elif kind == "dense":
        pos *= 0.05
    elif kind == "core":
        pos[: n // 8] *= 0.05
    return pos.astype(np.float32)


def handle(nb, pos, vel=None, algo=0):
    n = len(pos)
    s = nb.Simulation(num_of_bodies=n, algo_config=algo, collision=1, theta=0.7, gravitational_constant=0.0)
    s.set_state(pos, np.full(n, 1.0 / n, np.float32), vel)
    return s


# on both sides of the sizes that may have more left than the warps' form serves
# (256 bodies per SM: 38,912 on 152 SMs)
@pytest.mark.parametrize("kind,n", [("far", 5120), ("dense", 5120), ("core", 5121), ("core", 9999), ("far", 20011),
                                    ("core", 39003), ("far", 39003)])
@pytest.mark.parametrize("algo", [0, 2])
def test_fallbacks_bit_exact(gpu, oracle, kind, n, algo):
    if algo == 2 and n > 20011:
        pytest.skip("the tree system's order is the one that differs")
    nb = gpu
    pos = layout(kind, n)
    vel = (0.1 * np.random.default_rng(n + 1).normal(size=(n, 3))).astype(np.float32)
    with handle(nb, pos, vel, algo) as s:
        s.step(0.0, 1)  # no gravity, no drift: the collision update alone
        got = s.get_state()[1]
    np.testing.assert_array_equal(got, oracle.collision(pos, vel))


@pytest.mark.parametrize("kind", ["far", "dense", "core"])
def test_fallbacks_take_little_longer(gpu, kind):
    """5,119 bodies take the warp form (51 us, 400 the dense system); 5,120 the grid
    and what it leaves."""
    nb = gpu
    ms = []
    for n in (5119, 5120):
        with handle(nb, layout(kind, n)) as s:
            s.step(0.0, 1)
            s.set_profiling(True)
            took = []
            for _ in range(9):
                s.step(0.0, 1)
                took.append(s.timings()["collision"])
            ms.append(min(took))
    assert ms[1] < 3.0 * ms[0]


def cusp(n, inner=-4.0):
    """Half of the bodies within the contact distance of one another."""
    rng = np.random.default_rng(n)
    d = rng.normal(size=(n, 3))
    return (d / np.linalg.norm(d, axis=1)[:, None] * 10.0 ** rng.uniform(inner, 1, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("n,inner", [(5120, -4.0), (20011, -1.0), (38912, -1.5), (38913, -4.0)])
def test_cusp_bit_exact(gpu, oracle, n, inner):
    """Targets with thousands of contacts, and ones between those and the grid's."""
    pos = cusp(n, inner)
    vel = (0.1 * np.random.default_rng(n + 1).normal(size=(n, 3))).astype(np.float32)
    with handle(gpu, pos, vel) as s:
        s.step(0.0, 1)
        got = s.get_state()[1]
    np.testing.assert_array_equal(got, oracle.collision(pos, vel))


def test_thousands_of_contacts_take_the_block_form(gpu):
    """59,157 bodies of a cusp against as many in a ball with one far out, which
    all go through the blocks: their reflections take three times as long as all
    pair tests, a warp a target 25 times."""
    ms = []
    for pos in (layout("far", 59157), cusp(59157)):
        with handle(gpu, pos) as s:
            s.step(0.0, 1)
            s.set_profiling(True)
            took = []
            for _ in range(3):
                s.step(0.0, 1)
                took.append(s.timings()["collision"])
            ms.append(min(took))
    assert ms[1] < 8.0 * ms[0]


def test_all_in_contact_behind_the_direct_sums(gpu):
    """2,859 bodies, each in contact with all: the update is all there is to the step
    (0.64 ms of it) and takes a direct system what it takes a tree system."""
    pos = (1e-12 * np.random.default_rng(2859).uniform(-1, 1, (2859, 3))).astype(np.float32)
    ms = []
    for algo in (0, 1):
        with handle(gpu, pos, algo=algo) as s:
            s.step(0.0, 2)
            ms.append(min(s.time_steps(0.0, 4) for _ in range(6)))
    assert ms[1] < 1.2 * ms[0]
