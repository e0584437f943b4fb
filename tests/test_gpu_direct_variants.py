"""No launch shape of a batch's direct sum changes a result: a server runs every
variant there is and a batch's autotuner picks one by timing; the states are the
same bits each time.  Sizes around a tile of 64 bodies, a stream's eight tiles
and a block's targets."""
import numpy as np
import pytest

from test_gpu_batch import cfg

pytestmark = pytest.mark.gpu

SIZES = (1, 31, 64, 65, 511, 513, 1025, 4097)


def states():
    out = []
    for n in SIZES:
        rng = np.random.default_rng(n)
        mass = (rng.random(n) + 0.5).astype(np.float32)
        out.append((rng.normal(size=(n, 3)).astype(np.float32), mass / mass.sum(),
                    (0.05 * rng.normal(size=(n, 3))).astype(np.float32)))
    return out


def batched(nb, tune):
    with nb.Batch([cfg(nb, n, False, 3) for n in SIZES]) as b:
        for k, s in enumerate(states()):
            b.set_state(k, *s)
        if tune:
            b.autotune()
        b.step(1e-3, 3)
        return [b.get_state(k)[:2] for k in range(len(SIZES))]


def same(got, want):
    for k, (g, w) in enumerate(zip(got, want)):
        for a, r in zip(g, w):
            np.testing.assert_array_equal(a, r, err_msg=str(SIZES[k]))


def test_autotuned_batch(gpu):
    want = batched(gpu, False)
    for _ in range(3):
        same(batched(gpu, True), want)


@pytest.mark.parametrize("variant", range(11))
def test_served_variants(gpu, variant):
    nb = gpu
    with nb.Server(max_jobs=len(SIZES), snapshot_every=0, direct_variant=variant, numerical_method=nb.KDK_LEAPFROG) as s:
        ids = [s.submit(cfg(nb, n, False, 3), 3, 1e-3, *st) for n, st in zip(SIZES, states())]
        assert s.wait() == 0
        same([s.result(job, n) for job, n in zip(ids, SIZES)], batched(nb, False))


def test_cache_of_another_build(gpu, tmp_path):
    """Numbers that an earlier build wrote for its shapes name other kernels here:
    its entries are left alone and the batch is tuned."""
    import json

    nb = gpu
    cache = tmp_path / "tune.json"
    sizes = [(600, False), (3000, False), (5000, True)]

    def tune():
        with nb.Batch([cfg(nb, n, tree) for n, tree in sizes]) as b:
            for k, (n, _) in enumerate(sizes):
                rng = np.random.default_rng(n)
                b.set_state(k, rng.normal(size=(n, 3)).astype(np.float32), np.full(n, 1.0 / n, np.float32))
            b.autotune(str(cache))
        return json.loads(cache.read_text())

    sm = next(p for p in next(iter(tune())).split("/") if p.startswith("sm"))
    old = {f"batch_direct/{sm}/9x1/11x1": 10, f"batch_tree/{sm}/quad0/comp0/12x1": 107}
    cache.write_text(json.dumps(old))
    table = tune()
    assert len(table) == 4 and {k: table[k] for k in old} == old
