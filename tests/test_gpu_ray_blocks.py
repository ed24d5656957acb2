"""Ray queries where a block per ray can go wrong: equal distances (the lowest
body, and on a mesh the last triangle, wins), more crossed bodies than a
block's list holds, bodies and rays around a warp and a block, ignored bodies,
rays in the plane of a cylinder's cap; against the CPU restatement."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


def _both(sc):
    import oracle
    out = []
    for w in (cg.world(), oracle.port_world()):
        scenes.apply(sc, w)
        out.append(w)
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 65, 129, 700])
@pytest.mark.parametrize("rays", [1, 33, 1500])
def test_rays_along_a_row_of_bodies(n, rays):
    """A row of boxes and spheres: a ray along it crosses every one; all rays
    agree with the restatement on the body, the point and the distance."""
    sc = scenes.Scene("row", scenes.MIXED_PARAMS)
    for k in range(n):
        if k % 2:
            sc.sphere((0, 0, 0), 0.75, M, scenes.FIXED, (2.0 * k, 0, 0))
        else:
            sc.box((-.75, -.75, -.75), 1.5, 1.5, 1.5, M, scenes.FIXED, (2.0 * k, 0, 0))
    g, r = _both(sc)
    rng = np.random.default_rng(n + rays)
    o = np.zeros((rays, 3))
    o[:, 0] = np.where(np.arange(rays) % 2, -5.0, 2.0 * n + 5.0)
    o[:, 1:] = rng.uniform(-0.4, 0.4, (rays, 2))
    d = np.zeros((rays, 3))
    d[:, 0] = np.where(np.arange(rays) % 2, 1.0, -1.0)
    for ignore in ((), (1, n)):
        a, b = g.raycast(o, d, ignore), r.raycast(o, d, ignore)
        assert np.array_equal(a["body"], b["body"])
        assert np.allclose(a["dist"], b["dist"], rtol=1e-5, atol=1e-4)
        assert np.allclose(a["pos"], b["pos"], atol=1e-3)


def test_equal_distances_take_the_lowest_body():
    sc = scenes.Scene("twins", scenes.MIXED_PARAMS)
    for _ in range(40):
        sc.box((-1, -1, -1), 2.0, 2.0, 2.0, M, scenes.FIXED)
    g, r = _both(sc)
    o, d = np.array([[-4.0, 0.25, 0.5]]), np.array([[1.0, 0.0, 0.0]])
    for ignore in ((), (1, 2, 3)):
        assert g.raycast(o, d, ignore)["body"][0] == r.raycast(o, d, ignore)["body"][0] == (4 if ignore else 1)


def test_mesh_edges_and_cap_planes():
    """Rays onto the shared edges of a flat mesh (two triangles at one
    distance), and rays in the plane of a cylinder's cap."""
    h = np.zeros((9, 9))
    pts, tris = scenes.grid_mesh(h, 1.0, (-4.0, 0.0, -4.0))
    sc = scenes.Scene("flat", scenes.MIXED_PARAMS)
    sc.mesh(pts, tris, M)
    sc.cylinder((0.0, 2.0, 0.0), 0.5, 1.0, M, scenes.FIXED)
    g, r = _both(sc)
    xs = np.arange(-3.5, 3.6, 0.5)
    o = np.array([[x + 1.0, 5.0, z] for x in xs for z in xs if abs(x + 1.0) > 0.6 or abs(z) > 0.6])
    d = np.tile([0.0, -1.0, 0.0], (len(o), 1))
    a, b = g.raycast(o, d), r.raycast(o, d)
    assert np.array_equal(a["body"], b["body"]) and np.allclose(a["dist"], b["dist"], atol=1e-4)
    o = np.array([[-3.0, 3.0, 0.0], [-3.0, 2.0, 0.1], [-3.0, 2.5, 0.0]])
    d = np.tile([1.0, 0.0, 0.0], (3, 1))
    assert g.raycast(o, d)["body"][2] == 2
    again = g.raycast(o, d)
    assert np.array_equal(again["body"], g.raycast(o, d)["body"])
