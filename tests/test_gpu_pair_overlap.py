"""Allocation-free pair calls that overlap on two streams share their scratch, so
their pairs may be wrong; they still write nothing outside their buffers, end
without an error, and calls in order are right again afterwards."""
import ctypes

import numpy as np
import pytest

import constraintphysics_gb300 as cg

pytestmark = pytest.mark.gpu


def test_overlapping_calls_stay_in_their_buffers():
    torch = pytest.importorskip("torch")
    fn = cg.lib()._lib.cpgpu_pairs_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    rng = np.random.default_rng(1)
    calls, guard = [], 4096
    for n, spread, big in ((65536, 18.0, 0.0), (9001, 8.0, 0.3), (300, 3.0, 0.0), (20000, 6.0, 0.5)):
        c = rng.uniform(-spread, spread, (n, 3))
        h = rng.uniform(0.1, 0.6, (n, 3)) * np.where(rng.random((n, 1)) < big, 4.0, 1.0)
        cap = 4 * n
        calls.append((torch.from_numpy(np.concatenate([c - h, c + h], 1).astype(np.float32)).cuda(), n,
                      torch.full((cap + guard, 2), -1, dtype=torch.int32, device="cuda"), cap,
                      torch.zeros(1, dtype=torch.int32, device="cuda"), torch.cuda.Stream()))

    def call(k, stream):
        a, n, pairs, cap, count, _ = calls[k]
        assert fn(a.data_ptr(), n, pairs.data_ptr(), cap, count.data_ptr(), stream.cuda_stream) == 0

    want = []
    for k in range(len(calls)):   # in order on one stream
        call(k, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append((calls[k][2].cpu(), int(calls[k][4])))
    for _ in range(12):
        for k in range(len(calls)):
            call(k, calls[k][5])
    torch.cuda.synchronize()
    for _, _, pairs, cap, _, _ in calls:
        assert bool((pairs[cap:] == -1).all())
    for k in range(len(calls)):
        call(k, torch.cuda.current_stream())
        torch.cuda.synchronize()
        n = min(want[k][1], calls[k][3])
        assert int(calls[k][4]) == want[k][1]
        assert torch.equal(calls[k][2].cpu()[:n], want[k][0][:n])
