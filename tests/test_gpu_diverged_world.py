"""A world whose impulses overflow, among many others of a batch: the batch
reports it, and every other world gets the bits it has without that world.  The
solver's workers take many islands one after the other (4,000 islands here, at
most 1,520 workers), so what one island leaves behind in a worker would reach the
next: with the middling islands' workers (the default for 4 to 48 rows), with
the big ones' (every island big), and with velocity changes in global memory
(islands above 32 bodies)."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes
from constraintphysics_gb300.world import CPGPUError

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


def _resting(n, speed):
    """n cubes in a row on a plate, touching one another: one island; the last one falls with `speed`."""
    sc = scenes.Scene("rest", scenes.DROP_PARAMS)
    sc.box((-50.0, -1.0, -50.0), 100.0, 1.0, 100.0, M, scenes.FIXED)
    for k in range(n):
        b = sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, M, scenes.DYNAMIC, (0.999 * k, 0.4995, 0.0))
        sc.velocity(b, (0.1, -0.2 if k < n - 1 else -speed, 0.05))
    return sc


def _step(worlds, diverges):
    b = cg.Batch(worlds)
    if diverges:
        with pytest.raises(CPGPUError, match="non-finite-state"):
            b.step(1)
    else:
        b.step(1)
    return b.read_state().view(np.uint32)


@pytest.mark.parametrize("env,n,count", [({}, 1, 4000), ({"CPGPU_PGS_BIG_ROWS": "1"}, 1, 4000),
                                         ({"CPGPU_PGS_BIG_ROWS": "1", "CPGPU_PGS_DV_CAP": "32"}, 40, 600)])
def test_other_worlds_keep_their_bits(monkeypatch, env, n, count):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    own = []
    for speed in (0.3, 2e38):
        w = cg.world()
        scenes.apply(_resting(n, speed), w)
        own.append(w)
    bad = np.arange(count) % 5 == 2
    ref = _step([cg.clone(own[0]) for _ in range(count)], False).reshape(count, n + 1, 16)
    got = _step([cg.clone(own[int(x)]) for x in bad], True).reshape(count, n + 1, 16)
    assert (ref == ref[0]).all()
    assert not (got[bad] == ref[bad]).all()
    assert (got[~bad] == ref[~bad]).all()
