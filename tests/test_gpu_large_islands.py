"""Islands of worlds of more than 2,048 bodies without joints or sleeping: the
components searched beside each other (large ones by a warp, the others by a
thread, visits in shared memory or, above 40,960 bodies, in global memory)
against the one-thread search (CPGPU_ISLANDS_SERIAL=1).  The islands, rows and
row order are the same, so the states agree bit for bit."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


def _loose(n):
    """Rows of boxes on a plate, runs of 1 to 40 touching ones, some two high."""
    rng = np.random.default_rng(n)
    sc = scenes.Scene("loose", scenes.DROP_PARAMS)
    sc.box((-500.0, -1.0, -500.0), 1000.0, 1.0, 1000.0, scenes.PILE_MATERIAL, scenes.FIXED)
    k = row = 0
    while k < n:
        x = -300.0
        while k < n and x < 300.0:
            for _ in range(int(rng.integers(1, 41))):
                if k < n:
                    sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, scenes.PILE_MATERIAL, scenes.DYNAMIC, (x, 0.499, 2.5 * row - 300.0))
                    k += 1
                if k < n and rng.random() < 0.2:
                    sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, scenes.PILE_MATERIAL, scenes.DYNAMIC, (x, 1.498, 2.5 * row - 300.0))
                    k += 1
                x += 0.998
            x += 1.0
        row += 1
    return sc


def _scenes(kind):
    if kind == "loose_2048":   # with the plate one body above the line
        return [_loose(2048)], 6
    if kind == "loose_41000":
        return [_loose(41000)], 3
    if kind == "terrain":
        return [scenes.terrain_drop(1, 48, 16, 10)], 160
    pool = scenes.HullPool(1, size=32)
    rng = np.random.default_rng(3)
    return [scenes.batched_world(rng, pool, n + 0.5, n + 0.5) for n in (40, 2300, 2100, 300)], 80


@pytest.mark.parametrize("kind", ["loose_2048", "loose_41000", "terrain", "piles"])
def test_component_searches_equal_the_serial_search(monkeypatch, kind):
    got = []
    scs, steps = _scenes(kind)
    for serial in ("0", "1"):
        monkeypatch.setenv("CPGPU_ISLANDS_SERIAL", serial)
        worlds = []
        for sc in scs:
            w = cg.world()
            scenes.apply(sc, w)
            worlds.append(w)
        b = cg.Batch(worlds)
        out = []
        for _ in range(3):
            b.step(steps // 3)
            out.append(b.read_state().copy())
        got.append((np.stack(out), b.info()))
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0].view(np.uint32), got[1][0].view(np.uint32))
