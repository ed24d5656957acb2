"""A jointed world alone, whose joint rows are rebuilt by a lane of a warp each,
and as copies in a batch, where they fill the lanes: the same bits."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [60, 700])
@pytest.mark.parametrize("make", [scenes.heavy_chain, lambda: scenes.motor_chain(3, True), lambda: scenes.piston_chain(2),
                                  lambda: scenes.slider_chain(("slider", "sliding_hinge", "hinge", "slider"))],
                         ids=["ball", "motor", "piston", "slider"])
def test_a_jointed_world_alone_equals_its_copies(make, copies):
    out = []
    for n in (1, copies):
        w = cg.world()
        scenes.apply(make(), w)
        b = cg.Batch([w] + [cg.clone(w) for _ in range(n - 1)])
        b.step(40)
        out.append(b.read_state().reshape(n, -1))
    one = out[0].view(np.uint32)
    assert np.array_equal(np.broadcast_to(one, (copies, one.shape[1])), out[1].view(np.uint32))
