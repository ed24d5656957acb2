"""Candidate pairs at the sizes and boxes where the pair passes change: group
and chunk remainders, the line between the pass over all later boxes and the
hashed grid, boxes far larger than a cell, crowded cells, inverted and
non-finite boxes, boxes at unaligned addresses; against the overlap test in
numpy, exactly."""
import ctypes

import numpy as np
import pytest

import constraintphysics_gb300 as cg

pytestmark = pytest.mark.gpu


def _expected(a):
    """Pairs i < j (1-based, sorted) with no separating axis; comparisons with NaN separate nothing."""
    out = []
    for i in range(len(a) - 1):
        b = a[i + 1:]
        with np.errstate(invalid="ignore"):
            sep = ((a[i, 3:] < b[:, :3]) | (a[i, :3] > b[:, 3:])).any(axis=1)
        j = np.nonzero(~sep)[0] + i + 1
        out.append(np.stack([np.full(len(j), i), j], 1))
    return (np.concatenate(out) + 1).astype(np.uint32) if out else np.zeros((0, 2), np.uint32)


def _pairs(a, cap, shift=0):
    torch = pytest.importorskip("torch")
    fn = cg.lib()._lib.cpgpu_pairs_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    buf = torch.zeros(6 * len(a) + 4, dtype=torch.float32, device="cuda")
    buf[shift:shift + 6 * len(a)] = torch.from_numpy(a.reshape(-1)).cuda()
    pairs = torch.full((max(cap, 1), 2), -1, dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = fn(buf.data_ptr() + 4 * shift, len(a), pairs.data_ptr(), cap, count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, cg.lib().last_error()
    torch.cuda.synchronize()
    return pairs.cpu().numpy().view(np.uint32), int(count[0])


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1.0, 1.0, (n, 3)) * n ** (1 / 3) * 0.8
    h = rng.uniform(0.1, 0.6, (n, 3))
    if kind == "crowd":      # one crowded cell among the others
        c[: n // 20] *= 0.02
    a = np.concatenate([c - h, c + h], 1).astype(np.float32)
    if kind == "odd":        # plates, points, inverted, huge and non-finite boxes
        a[0] = [-500, -2, -500, 500, 0, 500]
        a[n // 2] = [-500, -500, 1, 500, 500, 1.5]
        a[3, 3:] = a[3, :3]
        a[5, [0, 3]] = a[5, [3, 0]]
        a[7] = np.nan
        a[9, 4] = np.inf
        a[11, 0] = -np.inf
        a[13, :] = 3e37
        a[15, 2] = np.nan
        a[n - 1] = [-1e7, -1e7, -1e7, 1e7, 1e7, 1e7]
    return a


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 5120, 5121, 9001])
@pytest.mark.parametrize("kind", ["plain", "crowd", "odd"])
def test_pairs_are_the_overlaps(n, kind):
    if kind == "odd" and n < 31:
        pytest.skip("too few boxes for the odd ones")
    a = _boxes(n, kind)
    want = _expected(a)
    got, count = _pairs(a, len(want) + 8, shift=n % 2)
    assert count == len(want)
    assert np.array_equal(got[:count], want)
    assert (got[count:].view(np.int32) == -1).all()


def test_count_beyond_capacity_writes_the_first_pairs_only():
    a = _boxes(6000, "odd")
    want = _expected(a)
    cap = len(want) // 2 + 1
    got, count = _pairs(a, cap)
    assert count == len(want)
    assert np.array_equal(got[:cap], want[:cap])
