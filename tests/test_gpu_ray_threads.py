"""Ray queries of several threads against one world at the same time: each gets
the hits of its own rays (the threads share the world's device buffer, which
grows with the largest query)."""
import threading

import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_queries_from_several_threads():
    w = cg.world()
    scenes.apply(scenes.mixed_drop(4, 5, n_layers=2), w)
    w.step(20)

    def rays(seed, n):
        rng = np.random.default_rng(seed)
        o = rng.uniform(-6.0, 6.0, (n, 3)) + np.array([0.0, 12.0, 0.0])
        d = rng.normal(size=(n, 3)) * np.array([0.3, 0.0, 0.3]) + np.array([0.0, -1.0, 0.0])
        return o, d / np.linalg.norm(d, axis=1, keepdims=True)

    # sizes that grow, each thread with its own
    jobs = [[rays(100 * t + k, 1 + 37 * t + 211 * k) for k in range(12)] for t in range(6)]
    alone, again = cg.clone(w), cg.clone(w)   # again's buffer has not grown yet
    want = [[alone.raycast(o, d) for o, d in job] for job in jobs]
    again.aabbs()
    bad, start = [], threading.Barrier(len(jobs))

    def work(t):
        start.wait()
        for rep in range(3):
            for (o, d), r in zip(jobs[t], want[t]):
                got = again.raycast(o, d)
                if any(not np.array_equal(got[k], r[k]) for k in ("body", "pos", "normal", "dist")):
                    bad.append((t, rep, len(o)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all((r["body"] > 0).any() for job in want for r in job[1:])
    assert not bad
