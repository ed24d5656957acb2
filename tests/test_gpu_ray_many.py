"""A call of many rays (a thread each) against calls of few (a block each): the
same hits, bit for bit, over hulls, round shapes, bodies of several primitives
and a mesh, with ignored bodies, rays from far away and non-finite ones."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: scenes.terrain_drop(1, 16, 4, 2), lambda: scenes.mixed_drop(2, 5, n_layers=2),
                                  lambda: scenes.union_drop(3, 12), lambda: scenes.capsule_drop(1, 3, 2, True)],
                         ids=["terrain", "mixed", "unions", "capsules"])
@pytest.mark.parametrize("n", [40960, 41023])
def test_many_rays_equal_few(make, n):
    w = cg.world()
    scenes.apply(make(), w)
    w.step(30)
    rng = np.random.default_rng(n)
    o = rng.uniform(-8.0, 8.0, (n, 3)) + np.array([0.0, 10.0, 0.0])
    o[::7] *= 30.0
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[5] = (0.0, -1.0, 0.0)
    o[11], d[13], o[17] = np.nan, np.nan, np.inf
    for ignore in ((), (2, 5, 6)):
        many = w.raycast(o, d, ignore)
        few = [w.raycast(o[k:k + 4096], d[k:k + 4096], ignore) for k in range(0, n, 4096)]
        assert (many["body"] > 0).mean() > 0.1
        for key in ("body", "pos", "normal", "dist"):
            assert np.array_equal(many[key], np.concatenate([f[key] for f in few]), equal_nan=many[key].dtype.kind == "f"), key
