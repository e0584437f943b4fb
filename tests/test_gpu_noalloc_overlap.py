"""Calls of nb_direct_accel_noalloc that overlap race on its shared scratch, as
its contract says; a later call that has it to itself gives the same bits as
before them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (777, 3001, 6007, 20001)  # different numbers of slices


def test_calls_after_an_overlap(gpu):
    torch = pytest.importorskip("torch")
    assert torch.cuda.is_available()
    L = gpu.load()
    bodies = [torch.randn(n, 4, device="cuda").abs() for n in SIZES]
    out = [torch.empty_like(b) for b in bodies]
    torch.cuda.synchronize()

    def call(k, acc, stream):
        return L.nb_direct_accel_noalloc(bodies[k].data_ptr(), SIZES[k], 0.01, 1.0, acc.data_ptr(), stream)

    def lone(k):
        out[k].fill_(-1.0)
        torch.cuda.synchronize()
        assert call(k, out[k], torch.cuda.current_stream().cuda_stream) == 0
        return out[k].cpu().numpy()

    want = [lone(k) for k in range(len(SIZES))]
    streams = [torch.cuda.Stream() for _ in SIZES]
    own = [torch.empty_like(b) for b in bodies]
    for _ in range(8):
        start = threading.Barrier(len(SIZES))
        status = [None] * len(SIZES)

        def run(k):
            start.wait()
            status[k] = [call(k, own[k], streams[k].cuda_stream) for _ in range(40)]

        threads = [threading.Thread(target=run, args=(k,)) for k in range(len(SIZES))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(s == [0] * 40 for s in status)
        for k in range(len(SIZES)):
            np.testing.assert_array_equal(lone(k), want[k], err_msg=str(SIZES[k]))
