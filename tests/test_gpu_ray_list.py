"""Rays that fill a block's list of crossed bodies again and again: every body
of a row is crossed, at sizes where the list (512 entries, 128 or 256 threads a
ray) is emptied after a full round, in the middle and at the end, with a mesh
among the listed bodies; against the CPU restatement.  Rays come from both ends,
and the nearest hit is once the first and once the last body listed, so a list
emptied early or read before it is complete loses it.  (Boxes: a plane's
distance is off by a few roundings of 1,500 m, 1e-3 m; a sphere's quadratic in
FP32 by up to its radius there.)"""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


@pytest.mark.parametrize("n", [256, 257, 384, 385, 511, 513, 640, 769, 1025])
@pytest.mark.parametrize("rays", [24, 1040])
def test_every_body_of_a_long_row_is_listed(n, rays):
    import oracle
    sc = scenes.Scene("row", scenes.MIXED_PARAMS)
    for k in range(n - 1):
        sc.box((-.6, -.6, -.6), 1.2, 1.2, 1.2, M, scenes.FIXED, (1.5 * k, 0, 0))
    pts = np.array([[1.5 * n, -3.0, -3.0], [1.5 * n, 3.0, -3.0], [1.5 * n, 0.0, 4.0]])
    sc.mesh(pts, np.array([[0, 1, 2]]), M)
    worlds = []
    for w in (cg.world(), oracle.port_world()):
        scenes.apply(sc, w)
        worlds.append(w)
    rng = np.random.default_rng(n)
    o, d = np.zeros((rays, 3)), np.zeros((rays, 3))
    o[:, 0] = np.where(np.arange(rays) % 2, -5.0, 1.5 * n + 5.0)
    o[:, 1:] = rng.uniform(-0.3, 0.3, (rays, 2))
    d[:, 0] = np.where(np.arange(rays) % 2, 1.0, -1.0)
    for ignore in ((), (n,), tuple(range(2, n + 1))):
        a, b = (w.raycast(o, d, ignore) for w in worlds)
        assert np.array_equal(a["body"], b["body"])
        assert np.allclose(a["dist"], b["dist"], rtol=1e-5, atol=1e-4)
        assert (a["body"] > 0).all()
