"""The warp's island search of a world in shared memory against the one-thread
search (CPGPU_ISLANDS_SERIAL=1): the same islands, rows and row order, so the
states agree bit for bit.  Worlds without contacts, of single bodies, of many
islands, of one, with kinematic and several fixed bodies, and sizes around a
warp and a block."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scenes(kind):
    rng = np.random.default_rng(7)
    pool = scenes.HullPool(1, size=32)
    if kind == "kinematic":
        return [scenes.kinematic_push(s) for s in range(3)]
    if kind == "drops":
        return [scenes.batched_world(rng, pool, n + 0.5, n + 0.5) for n in (1, 2, 8, 31, 32, 33, 64, 200, 257, 300)]
    out = []
    for n in (1, 40, 300):   # single bodies on two plates, some in the air, rows of touching boxes
        sc = scenes.Scene("loose", scenes.DROP_PARAMS)
        sc.box((-100.0, -1.0, -100.0), 200.0, 1.0, 100.0, scenes.PILE_MATERIAL, scenes.FIXED)
        sc.box((-100.0, -1.0, 0.0), 200.0, 1.0, 100.0, scenes.PILE_MATERIAL, scenes.FIXED)
        for k in range(n):
            gap = 0.995 if k % 7 < 4 else 1.7
            sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, scenes.PILE_MATERIAL, scenes.DYNAMIC,
                   (gap * (k % 30) - 15.0, 0.5 + (8.0 if k % 5 == 4 else 0.001), 2.0 * (k // 30) - 10.0))
        out.append(sc)
    return out


@pytest.mark.parametrize("kind", ["drops", "loose", "kinematic"])
def test_warp_search_equals_serial_search(monkeypatch, kind):
    got = []
    for serial in ("0", "1"):
        monkeypatch.setenv("CPGPU_ISLANDS_SERIAL", serial)
        worlds = []
        for sc in _scenes(kind):
            w = cg.world()
            scenes.apply(sc, w)
            worlds.append(w)
        b = cg.Batch(worlds)
        out = []
        for _ in range(60):
            b.step(2)
            out.append(b.read_state().copy())
        got.append((np.stack(out), b.info()))
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0].view(np.uint32), got[1][0].view(np.uint32))
