"""The region counts of the build from sorted paths are zero between steps,
whatever becomes of a step: a count left over would place bodies beyond their
region in the next one."""
import numpy as np
import pytest

from test_early_launch_loads import CSRC, kernels, source


def test_every_scan_block_clears_its_counts():
    """A wait for another block's total that gives up (2^24 polls of a running
    block) cannot be brought about, so its path is read from the source: no block
    of k_scan returns before its counts are published and cleared."""
    body = dict(kernels(source(CSRC + "/k_build.cu")))["k_scan"]
    assert "return" not in body.replace("return c0.x", "")
    assert body.index("st_volatile(&b.total[place]") < body.index("set_status") < body.index("int4(0, 0, 0, 0);\n        }")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2049, 20000, 300001])
def test_steps_after_failed_ones(gpu, n):
    nb = gpu
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)).astype(np.float32)
    mass = np.full(n, 1.0 / n, np.float32)
    bad = pos.copy()
    bad[n // 2, 1] = np.nan
    cfg = dict(num_of_bodies=n, algo_config=nb.BARNES_HUT, theta=0.7, epsilon=0.01, gravitational_constant=1.0)
    with nb.Simulation(**cfg) as fresh:
        fresh.set_state(pos, mass)
        fresh.step(1e-3, 2)
        want = fresh.get_state()
    with nb.Simulation(**cfg) as s:
        s.set_state(bad, mass)
        assert s.step(1e-3, 3, check=False) == nb.ERR_NONFINITE
        s.set_state(pos, mass)
        s.set_spin_cap(1 << 20)  # builds by insertions
        s.step(0.0, 1)
        s.set_spin_cap(0)
        s.set_state(pos, mass)
        s.step(1e-3, 2)
        for got, w in zip(s.get_state(), want):
            np.testing.assert_array_equal(got, w)


def test_large_reference_sort_waits_for_nobody():
    """The sort of large trees with the reference's semantics (k_tree.cu) runs on a
    plain grid, whose blocks may start in any order and late: no loop of it waits
    for what another thread writes (a bounded climb to the root is all there is)."""
    called = "sort_cell"
    assert called in dict(kernels(source(CSRC + "/k_tree.cu")))["k_sort"]
    device = source(CSRC + "/bh_device.cuh")
    at = device.index(f" {called}(const DevSim")
    function = device[at:device.index("\n}\n", at)]
    assert "__nanosleep" not in function and "while" not in function and "spin" not in function.lower().replace("kstspintimeout", "")
