"""Prefixes over many items (bodies, pairs, edges, contacts, islands) at the
sizes where the one-launch scan changes: below, at and above a chunk (2,048
items), and beyond 32 chunks (the look-back's window).  Every copy of a world
in a batch steps exactly as the world alone."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 255, 256, 257, 1025, 9000])
def test_every_copy_steps_as_the_world_alone(copies):
    sc = scenes.Scene("stack", scenes.DROP_PARAMS)
    sc.box((-10.0, -1.0, -10.0), 20.0, 1.0, 20.0, scenes.PILE_MATERIAL, scenes.FIXED)
    rng = np.random.default_rng(3)
    for k in range(7):   # with the plate 8 bodies, two stacks touching
        b = sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, scenes.PILE_MATERIAL, scenes.DYNAMIC,
                   (0.995 * (k % 2), 0.51 + 1.003 * (k // 2), 0.02 * k))
        sc.velocity(b, tuple(rng.uniform(-0.3, 0.3, 3)))
    w = cg.world()
    scenes.apply(sc, w)
    alone = cg.Batch([cg.clone(w)])
    b = cg.Batch([cg.clone(w) for _ in range(copies)])
    for steps in (1, 6, 14):
        alone.step(steps)
        b.step(steps)
        want = alone.read_state().view(np.uint32)
        got = b.read_state().view(np.uint32).reshape(copies, 8, 16)
        assert np.array_equal(got, np.broadcast_to(want, got.shape))
    assert b.info()["contacts"] == copies * alone.info()["contacts"] > 0
