"""The build from sorted octant paths against the oracle: sizes around a tile
of 256 bodies and around the switch from ranking all bodies to ranking regions,
crowded regions and bodies far out (the insertions take over), bodies that 21
levels do not part, and cells that reach over many tiles.  Topology, sort, cell
sums and counts are bit-exact."""
import numpy as np
import pytest

from test_gpu_parity import bh_sim, cell_table

pytestmark = pytest.mark.gpu


def bodies(kind, n):
    rng = np.random.default_rng(n + len(kind))
    pos = rng.normal(size=(n, 3)) if kind != "ball" else rng.uniform(-1, 1, (n, 3))
    if kind == "clumps":  # a few dense clumps: deep chains of cells, wide cells over many tiles
        pos = pos * 1e-3 + rng.integers(-2, 3, (n, 3))
    elif kind == "outlier":  # nearly all bodies in one region
        pos[0] = (4000.0, -3000.0, 2000.0)
    elif kind == "close":  # a pair that parts below level 21
        pos *= 1e-3
        pos[0] = (64.0, 64.0, 64.0)
        pos[n // 2] = pos[n // 3]
        pos[n // 2, 0] = np.nextafter(np.float32(pos[n // 3, 0]), np.float32(10))
    elif kind == "plane":
        pos[:, 2] = 0.25
    mass = (rng.random(n) + 0.5).astype(np.float32)
    return pos.astype(np.float32), mass / mass.sum()


SIZES = [("ball", n) for n in (1, 2, 3, 255, 256, 257, 511, 1025, 2047, 2048, 2049, 8193, 40000)]
KINDS = [("clumps", 3000), ("clumps", 30001), ("outlier", 5000), ("outlier", 60001), ("close", 700), ("close", 20000),
         ("plane", 10007)]


@pytest.mark.parametrize("kind,n", SIZES + KINDS)
@pytest.mark.parametrize("quad", [0, 1])
def test_tree_against_oracle(gpu, oracle, kind, n, quad):
    nb = gpu
    pos, mass = bodies(kind, n)
    sim = bh_sim(nb, pos, mass, 0.6, 0.01, quad=quad)
    for _ in range(2):  # the second step sees what the first one left in the tables
        assert sim.step(0.0, 1, check=False) == 0
    info = sim.stage_debug(nb.DEBUG_TREE_INFO)
    cap = int(info[1])
    t = oracle.tree_build(oracle.SEM_GEOMETRIC, pos, mass, sim.stage_debug(nb.DEBUG_BBOX), cap)
    assert t.status == 0 and int(info[2]) == t.bottom
    assert max(int(info[3]), 1) == t.max_depth  # the oracle counts from 1 (a body under the root is at 0 here)
    children = sim.stage_debug(nb.DEBUG_CHILDREN)
    pg, dg, fg = oracle.tree_paths(children, n, n + cap)
    po, do, fo = oracle.tree_paths(t.children, n, t.root)
    assert fg == n and fo == n and np.array_equal(dg, do) and np.array_equal(pg, po)
    octant = t.children.copy()
    assert oracle.saturate(t) == 0
    tg = cell_table(children, sim.stage_debug(nb.DEBUG_NODE_MASS), sim.stage_debug(nb.DEBUG_NODE_POS),
                    sim.stage_debug(nb.DEBUG_BODY_COUNT), n, n + cap)
    to = cell_table(octant, t.mass, t.pos, t.body_count, n, t.root)
    assert tg == to
    order, k = oracle.sort_bodies(t.children, n, t.root)
    assert k == n and np.array_equal(sim.stage_debug(nb.DEBUG_SORTED), order)
    if quad:
        qg = sim.stage_debug(nb.DEBUG_NODE_QUAD).reshape(-1, 6)
        qo = oracle.quadrupoles(t).reshape(-1, 6)
        zero = np.zeros(len(qg))
        ig = cell_table(children, zero, np.zeros((len(qg), 3)), np.arange(len(qg)), n, n + cap)
        io = cell_table(octant, np.zeros(len(qo)), np.zeros((len(qo), 3)), np.arange(len(qo)), n, t.root)
        for path in io:
            assert np.array_equal(qg[ig[path][2]], qo[io[path][2]]), path
    # the walk on this tree
    acc = oracle.bh_step_forces(pos, mass, 0.6, 0.01, 1.0, nodes=cap, quadrupole=bool(quad))[0]
    scale = np.sqrt(np.mean(np.sum(acc.astype(np.float64) ** 2, axis=1)))
    assert np.max(np.linalg.norm(sim.get_state()[2] - acc.astype(np.float64), axis=1)) <= 2e-5 * scale


@pytest.mark.parametrize("n", [5000, 6500, 11000, 12500, 14000, 32768, 32769])
@pytest.mark.parametrize("quad", [0, 1])
def test_lists_around_the_one_block_form(gpu, oracle, n, quad):
    """Trees whose cells over a tile's edge are about as many as one block takes."""
    test_tree_against_oracle(gpu, oracle, "ball", n, quad)


@pytest.mark.parametrize("kind,n", [("ball", n) for n in (1, 2, 257, 2048, 2049, 20000, 131072, 131073)] +
                         [("clumps", 3000), ("outlier", 5000), ("close", 700), ("plane", 10007)])
@pytest.mark.parametrize("quad", [0, 1])
def test_reference_tree_against_oracle(gpu, oracle, kind, n, quad):
    """The reference's boxes and super-root, from paths and, beyond 131,072 bodies
    or where paths do not part them, from insertions."""
    nb = gpu
    pos, mass = bodies(kind, n)
    if kind == "close":  # the reference's boxes part bodies along x and z
        pos[n // 2] += np.float32(1e-4)
    sim = bh_sim(nb, pos, mass, 0.6, 0.01, tree=1, quad=quad)
    for _ in range(2):
        assert sim.step(0.0, 1, check=False) == 0
    info = sim.stage_debug(nb.DEBUG_TREE_INFO)
    cap = int(info[1])
    t = oracle.tree_build(oracle.SEM_REFERENCE, pos, mass, sim.stage_debug(nb.DEBUG_BBOX), cap)
    assert t.status == 0 and int(info[2]) == t.bottom
    children = sim.stage_debug(nb.DEBUG_CHILDREN)
    pg, dg, fg = oracle.tree_paths(children, n, n + cap)
    po, do, fo = oracle.tree_paths(t.children, n, t.root)
    assert fg == n and fo == n and np.array_equal(dg, do) and np.array_equal(pg, po)
    octant = t.children.copy()
    assert oracle.saturate(t) == 0
    tg = cell_table(children, sim.stage_debug(nb.DEBUG_NODE_MASS), sim.stage_debug(nb.DEBUG_NODE_POS),
                    sim.stage_debug(nb.DEBUG_BODY_COUNT), n, n + cap)
    assert tg == cell_table(octant, t.mass, t.pos, t.body_count, n, t.root)
    order, k = oracle.sort_bodies(t.children, n, t.root)
    assert k == n and np.array_equal(sim.stage_debug(nb.DEBUG_SORTED), order)


@pytest.mark.parametrize("quad", [0, 1])
def test_large_tree_against_oracle(gpu, oracle, quad):
    """From 2^20 bodies the upper cells' kernel has twice the threads."""
    test_tree_against_oracle(gpu, oracle, "ball", (1 << 20) + 1, quad)
