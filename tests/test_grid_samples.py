"""The boxes that size the pair grid's cells: at most 4,096, evenly spaced over
all boxes of the grid, whatever their number and wherever the large worlds of a
batch stand."""
import os
import subprocess

import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

HERE = os.path.dirname(os.path.abspath(__file__))


def test_samples_cover_all_boxes_of_the_grid(tmp_path):
    exe = str(tmp_path / "grid_samples")
    csrc = os.path.join(os.path.dirname(cg.__file__), "csrc")
    subprocess.run(["g++", "-std=c++17", "-I" + csrc, os.path.join(HERE, "cxx", "grid_samples.cpp"), "-o", exe], check=True)
    lines = [[int(x) for x in line.split()] for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split("\n") if line]
    for n, m, last, step in (x for x in lines if len(x) == 4):
        assert 1 <= m <= 4096 and last < n <= last + step
        assert m > min(n, 4096) / 2
    picked = np.array([x[0] for x in lines if len(x) == 1])
    want = np.concatenate([np.arange(5200, 7300), np.arange(7420, 10420)])   # the bodies of the two large worlds
    step = -(-len(want) // 4096)
    assert np.array_equal(picked, want[::step])


@pytest.mark.gpu
def test_large_world_behind_many_small_ones():
    """The large world's bodies all come after 5,200 bodies of small worlds; it steps as it does alone."""
    pool = scenes.HullPool(1, size=32)
    rng = np.random.default_rng(11)
    big, small = scenes.batched_world(rng, pool, 2300.5, 2300.5), scenes.batched_world(rng, pool, 40.5, 40.5)
    own = []
    for sc in (small, big):
        w = cg.world()
        scenes.apply(sc, w)
        own.append(w)
    n = own[1].n_bodies
    alone = cg.Batch([cg.clone(own[1])])
    among = cg.Batch([cg.clone(own[0]) for _ in range(130)] + [own[1]])
    for b in (alone, among):
        b.step(40)
    assert np.array_equal(alone.read_state().view(np.uint32), among.read_state()[-n:].view(np.uint32))
