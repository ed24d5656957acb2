"""The warp-per-island solver chain (rows resident in shared memory, rows
streamed through it, velocity changes in shared or global memory) against the
thread-per-island solver: the two run the same rows in the same order with the
same rounding, so the states agree bit for bit.  Sizes around the ring's
limits: islands of one contact, of a chunk (32 rows), of the resident limit
(96 rows) and beyond."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


def _stack_world(n, seed):
    """n boxes in wobbling columns touching each other: one island of about
    4 rows per touching pair (sliding and sticking contacts)."""
    rng = np.random.default_rng(seed)
    sc = scenes.Scene("stack", dict(scenes.DROP_PARAMS, pgs=(7, 2, 1)))
    sc.box((-20.0, -1.0, -20.0), 40.0, 1.0, 40.0, scenes.PILE_MATERIAL, scenes.FIXED)
    side = max(1, int(round(n ** (1.0 / 3.0))))
    for k in range(n):
        x, z, y = k % side, k // side % side, k // (side * side)
        b = sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, scenes.PILE_MATERIAL, scenes.DYNAMIC,
                   (0.99 * x + rng.uniform(-.02, .02), 0.51 + 1.003 * y, 0.99 * z + rng.uniform(-.02, .02)))
        sc.velocity(b, tuple(rng.uniform(-0.4, 0.4, 3)))
    return sc


def _run(monkeypatch, sizes, steps, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, str(v))
    worlds = []
    for i, n in enumerate(sizes):
        w = cg.world()
        scenes.apply(_stack_world(n, i), w)
        worlds.append(w)
    b = cg.Batch(worlds)
    out = []
    for _ in range(steps):
        b.step(1)
        out.append(b.read_state().copy())
    return np.stack(out), b.info()["contacts"]


@pytest.mark.parametrize("sizes", [(1, 2, 3), (4, 5, 7, 8, 9), (12, 16, 24, 27), (40, 64, 90)])
def test_chain_solver_equals_thread_solver(monkeypatch, sizes):
    ref, contacts = _run(monkeypatch, sizes, 25, CPGPU_PGS_BIG_ROWS=1 << 30)
    assert contacts > 0
    got, _ = _run(monkeypatch, sizes, 25, CPGPU_PGS_BIG_ROWS=1)
    assert np.array_equal(ref.view(np.uint32), got.view(np.uint32))


def test_chain_solver_with_velocity_changes_in_global_memory(monkeypatch):
    sizes = (20, 40, 90)   # islands on both sides of the 32-body shared area
    ref, _ = _run(monkeypatch, sizes, 25, CPGPU_PGS_BIG_ROWS=1 << 30)
    got, _ = _run(monkeypatch, sizes, 25, CPGPU_PGS_BIG_ROWS=1, CPGPU_PGS_DV_CAP=32)
    assert np.array_equal(ref.view(np.uint32), got.view(np.uint32))
