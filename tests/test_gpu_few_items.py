"""One world stepped alone and as copies in a batch: alone its pairs and edges
are few enough for a warp each in the clip and the contact merge, and its island
pass takes 1,024 threads above 256 bodies; the batch of copies takes a thread per
pair and 256 threads a world.  Every copy's states are the same bits."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies,copies", [(1, 160), (12, 400), (255, 40), (257, 160), (400, 153)])
def test_a_world_alone_equals_its_copies(bodies, copies):
    rng = np.random.default_rng(bodies)
    sc = scenes.batched_world(rng, scenes.HullPool(2, size=16), bodies + 0.5, bodies + 0.5)
    out = []
    for n in (1, copies):
        w = cg.world()
        scenes.apply(sc, w)
        b = cg.Batch([w] + [cg.clone(w) for _ in range(n - 1)])
        b.step(60)
        out.append(b.read_state().reshape(n, -1))
    one = out[0].view(np.uint32)
    assert np.array_equal(np.broadcast_to(one, (copies, one.shape[1])), out[1].view(np.uint32))
