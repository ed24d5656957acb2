"""Worlds whose contact graph just fits shared memory: with the search's lists
beside it, only without them, or not at all; and batches of many tiny worlds,
whose islands smaller blocks search.  Against the one-thread search
(CPGPU_ISLANDS_SERIAL=1): the same islands and row order, so the same bits."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


def _packed(n, layers=11):
    """n touching spheres in a block: about 2.8 edges a body."""
    sc = scenes.Scene("packed", dict(scenes.DROP_PARAMS, pgs=(2, 1, 1)))
    sc.box((-200.0, -1.0, -200.0), 400.0, 1.0, 400.0, M, scenes.FIXED)
    side = int(np.ceil((n / layers) ** 0.5))
    for k in range(n):
        y, r = divmod(k, side * side)
        b = sc.sphere((0, 0, 0), 0.5, M, scenes.DYNAMIC, (0.9995 * (r % side), 0.4995 + 0.999 * y, 0.9995 * (r // side)))
        sc.velocity(b, (0.0, 0.0, 0.01 * (k % 7)))
    return sc


def _equal(monkeypatch, make, steps):
    got = []
    for serial in ("0", "1"):
        monkeypatch.setenv("CPGPU_ISLANDS_SERIAL", serial)
        b = cg.Batch(make())
        out = []
        for _ in range(steps):
            b.step(1)
            out.append(b.read_state().copy())
        got.append((np.stack(out).view(np.uint32), b.info()))
    assert got[0][1] == got[1][1] and got[0][1]["contacts"] > 0
    assert (got[0][0] == got[1][0]).all()


@pytest.mark.parametrize("sizes", [(1440,), (1480,), (1560,), (1640,), (300, 1500, 40, 1520)])
def test_graphs_around_the_size_of_shared_memory(monkeypatch, sizes):
    def make():
        worlds = []
        for n in sizes:
            w = cg.world()
            scenes.apply(_packed(n), w)
            worlds.append(w)
        return worlds
    _equal(monkeypatch, make, 6)


@pytest.mark.parametrize("copies", [600, 620, 3000])
def test_many_tiny_worlds(monkeypatch, copies):
    pool = scenes.HullPool(1, size=32)

    def make():
        own = []
        for k in range(12):
            w = cg.world()
            scenes.apply(scenes.batched_world(np.random.default_rng(k), pool, 2.5 + 5 * k, 2.5 + 5 * k), w)
            own.append(w)
        return own + [cg.clone(own[k % 12]) for k in range(12, copies)]
    _equal(monkeypatch, make, 30)
