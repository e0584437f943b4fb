"""State transfers with the host arrays a caller may hand over: ones that are
not aligned as floats (slices of a packed buffer) and managed memory, both of
which go through the staging, and memory that nothing has touched yet.  What is
set is what comes back, bit for bit."""
import ctypes
import mmap
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1029


def shifted(shape, by, src=None):
    """A float32 array `by` bytes behind an aligned address."""
    count = int(np.prod(shape))
    raw = np.zeros(4 * count + 64, np.uint8)
    at = (-raw.ctypes.data) % 16 + by
    a = raw[at:at + 4 * count].view(np.float32).reshape(shape)
    assert a.ctypes.data % 16 == by
    if src is not None:
        a[...] = src
    return a


def state(n=N):
    rng = np.random.default_rng(n)
    return (rng.normal(size=(n, 3)).astype(np.float32), rng.normal(size=(n, 3)).astype(np.float32),
            (rng.random(n) + 0.5).astype(np.float32))


def arrays(make):
    return [make((N, 3)), make((N, 3)), make((N, 3)), make((N,))]


def round_trip(nb, make):
    """Through a handle and through a batch; `make` gives the arrays."""
    pos, vel, mass = state()
    p, v, m = make((N, 3)), make((N, 3)), make((N,))
    p[...], v[...], m[...] = pos, vel, mass
    zero = np.zeros((N, 3), np.float32)
    with nb.Simulation(num_of_bodies=N, algo_config=nb.BRUTE_FORCE_LOCAL) as s:
        assert s.L.nb_set_state(s.h, p.ctypes.data, v.ctypes.data, m.ctypes.data, N) == 0
        for got, want in zip(s.get_state(), (pos, vel, zero, mass)):
            np.testing.assert_array_equal(got, want)
        out = arrays(make)
        assert s.L.nb_get_state(s.h, *(a.ctypes.data for a in out)) == 0
        for got, want in zip(out, (pos, vel, zero, mass)):
            np.testing.assert_array_equal(got, want)
        assert s.L.nb_set_state(s.h, p.ctypes.data, None, m.ctypes.data, N) == 0
        np.testing.assert_array_equal(s.get_state()[1], zero)
    c = nb.default_config(num_of_bodies=N, algo_config=nb.BRUTE_FORCE_LOCAL, epsilon=0.01)
    with nb.Batch([c, c]) as b:
        assert b.L.nb_batch_set_state(b.h, 1, p.ctypes.data, v.ctypes.data, m.ctypes.data) == 0
        for got, want in zip(b.get_state(1), (pos, vel, zero, mass)):
            np.testing.assert_array_equal(got, want)
        out = arrays(make)
        assert b.L.nb_batch_get_state(b.h, 1, *(a.ctypes.data for a in out)) == 0
        for got, want in zip(out, (pos, vel, zero, mass)):
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("by", [0, 1, 2, 3, 4])
def test_any_address(gpu, by):
    round_trip(gpu, lambda shape: shifted(shape, by))


def test_managed_memory(gpu):
    """Neither page-locked nor ordinary memory: the staging takes it."""
    torch = pytest.importorskip("torch")
    assert torch.cuda.is_available()
    torch.zeros(1, device="cuda")
    cuda = ctypes.CDLL("libcuda.so.1")
    held = []

    def make(shape):
        ptr = ctypes.c_uint64(0)
        size = 4 * int(np.prod(shape))
        assert cuda.cuMemAllocManaged(ctypes.byref(ptr), ctypes.c_size_t(size), ctypes.c_uint(1)) == 0
        held.append(ptr.value)
        buf = (ctypes.c_float * (size // 4)).from_address(ptr.value)
        a = np.frombuffer(buf, np.float32).reshape(shape)
        a[...] = 0.0
        return a

    try:
        round_trip(gpu, make)
    finally:
        torch.cuda.synchronize()
        for p in held:
            cuda.cuMemFree_v2(ctypes.c_uint64(p))


def time_of(read):
    t = time.perf_counter()
    read()
    return time.perf_counter() - t


def test_untouched_memory(gpu):
    """Large arrays whose pages the host never touched (an output array's first
    use) cost a few times the transfer into pages that are there, not fifty times:
    the pages are populated many at a time, not one fault of the device each."""
    nb = gpu
    n = 2000003
    pos, vel, mass = state(n)
    with nb.Simulation(num_of_bodies=n, algo_config=nb.BRUTE_FORCE_LOCAL) as s:
        s.set_state(pos, mass, vel)
        touched = np.ones((n, 3), np.float32)
        s.positions(out=touched)
        there, first = [], []
        for _ in range(5):
            there.append(time_of(lambda: s.positions(out=touched)))
            m = mmap.mmap(-1, 12 * n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
            fresh = np.frombuffer(m, np.float32).reshape(n, 3)
            first.append(time_of(lambda: s.positions(out=fresh)))
            np.testing.assert_array_equal(fresh, pos)
        # 24 MB into pages that are there 0.15 ms; populated first 0.9 ms, by
        # faults 7 ms
        assert min(first) < 20 * min(there)
        # untouched inputs read as zeros
        m = mmap.mmap(-1, 12 * n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
        s.set_state(pos, mass, np.frombuffer(m, np.float32).reshape(n, 3))
        assert not s.positions(with_velocities=True)[1].any()
