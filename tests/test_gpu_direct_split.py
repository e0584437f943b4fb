"""The direct sum where its split has edges: sizes around a lane's pair, a
tile and a target set, sizes that take several slices of the bodies, and the
allocation-free form writing over its own input."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n):
    rng = np.random.default_rng(n)
    m = (rng.random(n) + 0.5).astype(np.float32)
    return rng.normal(size=(n, 3)).astype(np.float32), (m / m.sum()).astype(np.float32)


def error(a, b):
    return np.max(np.linalg.norm(a.astype(np.float64) - b, axis=1)) / np.sqrt(np.mean(np.sum(b.astype(np.float64) ** 2, axis=1)))


# 2e-5 of the typical |a|: FP32 sums in two orders, each term within 1e-6
@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 64, 65, 127, 511, 513, 2047, 8191, 20001])
@pytest.mark.parametrize("algo,eps", [(1, 0.05), (2, 0.05), (1, 0.0), (2, 0.0)])
def test_sizes_against_oracle(gpu, oracle, n, algo, eps):
    pos, mass = system(n)
    sim = gpu.Simulation(num_of_bodies=n, algo_config=algo, direct_epsilon=eps, gravitational_constant=1.0)
    sim.set_state(pos, mass)
    runs = []
    for _ in range(2):  # the second step sees the counters the first one left
        sim.step(0.0, 1)
        runs.append(sim.get_state()[2])
    assert np.array_equal(runs[0], runs[1])
    want = oracle.direct_fp64(pos, mass, eps, 1.0) if eps == 0.0 else oracle.direct_fp32(pos, mass, eps, 1.0)
    if n == 1:
        assert np.all(runs[0] == 0.0)
    else:
        assert error(runs[0], want) < 2e-5


@pytest.mark.parametrize("n", [97, 3001])
def test_accelerations_over_the_bodies(gpu, n):
    import torch
    pos, mass = system(n)
    body = torch.from_numpy(np.concatenate([pos, mass[:, None]], 1)).cuda().contiguous()
    out = torch.empty_like(body)
    L = gpu.load()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.nb_direct_accel_noalloc(body.data_ptr(), n, 0.05, 1.0, out.data_ptr(), stream) == 0
    assert L.nb_direct_accel_noalloc(body.data_ptr(), n, 0.05, 1.0, body.data_ptr(), stream) == 0
    a, b = out.cpu().numpy()[:, :3], body.cpu().numpy()[:, :3]
    assert error(b, a) < 2e-6  # the same sums in one slice
