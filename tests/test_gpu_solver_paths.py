"""The solver's three paths -- a thread an island, a warp with the island's rows
in 21 KB of shared memory (4 to 48 rows), a warp that streams or holds larger
ones -- on islands of the same rows at the paths' limits: the states agree bit
for bit."""
import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


def _island(rows):
    """One island of exactly `rows` contacts at the first step: spheres in a row on a
    plate, each touching the plate and the next one (2 n - 1), and for an even
    number one more lying against the first alone."""
    rng = np.random.default_rng(rows)
    sc = scenes.Scene("island", dict(scenes.DROP_PARAMS, pgs=(7, 3, 1), substeps=2))
    sc.box((-100.0, -1.0, -100.0), 200.0, 1.0, 200.0, M, scenes.FIXED)
    n = (rows + 1) // 2
    ids = [sc.sphere((0, 0, 0), 0.5, M, scenes.DYNAMIC, (0.998 * k, 0.499, 0.0)) for k in range(n)]
    if rows % 2 == 0:
        ids.append(sc.sphere((0, 0, 0), 0.5, M, scenes.DYNAMIC, (-0.7, 1.2, 0.0)))
    for b in ids:
        sc.velocity(b, tuple(rng.uniform(-0.3, 0.3, 3)))
        sc.ang_velocity(b, tuple(rng.uniform(-0.5, 0.5, 3)))
    return sc


@pytest.mark.parametrize("rows", [(1, 2, 3, 4, 5), (15, 16, 17), (31, 32, 33), (47, 48, 49), (95, 96, 97)])
def test_three_paths_give_the_same_bits(monkeypatch, rows):
    got = []
    for big_rows in (1 << 30, 98, 1):   # a thread each; the middling class up to 48 rows; a warp each
        monkeypatch.setenv("CPGPU_PGS_BIG_ROWS", str(big_rows))
        worlds = []
        for r in rows:
            w = cg.world()
            scenes.apply(_island(r), w)
            worlds.append(w)
        b = cg.Batch(worlds)
        out = []
        for k in range(15):
            b.step(1)
            if k == 0:
                assert b.info()["contacts"] == sum(rows)
            out.append(b.read_state().copy())
        got.append(np.stack(out).view(np.uint32))
    assert (got[0] == got[1]).all()
    assert (got[0] == got[2]).all()
