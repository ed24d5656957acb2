"""Jointed islands past what a solver warp holds in shared memory (64 joint rows,
68 bodies, 128 rows in all; systems of 64 constraints and 96 blocks below the
diagonal; 40 KB of factor): longer chains, a chain lying on a plate, a hub with
many arms, in FP64 (mass ratios above 100) and FP32; against the restatement, a
step at a time from the same state, within the bounds of the shorter chains.  And
islands held in shared memory against the same islands in global memory
(CPGPU_PGS_DV_CAP=32), bit for bit."""
import math

import numpy as np
import pytest

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

pytestmark = pytest.mark.gpu
M = scenes.PILE_MATERIAL


def _link(sc, rng, heavy, pos):
    b = sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, M, scenes.DYNAMIC, pos)
    top = 100.0 if heavy else 5.0
    sc.mass(b, float(math.exp(rng.uniform(math.log(top / (1000.0 if heavy else 20.0)), math.log(top)))))
    return b


def _chain(n, heavy, y=0.0, plate=False):
    """n links in a line, ball-sockets and hinges in turn: hung at one end, or lying on a plate."""
    rng = np.random.default_rng(n + heavy)
    sc = scenes.Scene("chain_%d" % n, scenes.CHAIN_PARAMS)
    if plate:
        sc.box((-200.0, -1.5, -200.0), 400.0, 1.0, 400.0, M, scenes.FIXED)
        prev = None
    else:
        prev = sc.box((-0.5, -0.5, -0.5), 1.0, 1.0, 1.0, M, scenes.FIXED)
    for i in range(n):
        b = _link(sc, rng, heavy, (1.1 * (i + 1), -0.002 if plate else 0.0, 0.0))
        if prev is not None:
            a = (0.55, 0.0, 0.0), (-0.55, 0.0, 0.0)
            if i % 2 == 0:
                sc.ball_socket(prev, b, *a)
            else:
                axis = tuple(scenes.unit_sphere_points(rng, 1)[0])
                sc.hinge(prev, b, *a, axis, axis)
        prev = b
    return sc


def _hub(n, heavy):
    """A hub with n arms of two links: the arms' first joints all share a body."""
    rng = np.random.default_rng(n)
    sc = scenes.Scene("hub_%d" % n, scenes.CHAIN_PARAMS)
    post = sc.box((-0.5, 4.5, -0.5), 1.0, 1.0, 1.0, M, scenes.FIXED)
    hub = sc.sphere((0, 0, 0), 2.0, M, scenes.DYNAMIC)
    sc.mass(hub, 100.0 if heavy else 20.0)
    sc.ball_socket(post, hub, (0.0, 4.5, 0.0), (0.0, 4.5, 0.0))
    for k in range(n):
        c, s = math.cos(2 * math.pi * k / n), math.sin(2 * math.pi * k / n)
        prev, r0 = hub, 0.0
        for r in (5.0, 7.0):
            b = sc.sphere((0, 0, 0), 0.4, M, scenes.DYNAMIC, (r * c, 0.0, r * s))
            sc.mass(b, 0.5 if heavy else 2.0)
            at = 0.5 * (r0 + r) if r0 else 2.5
            sc.ball_socket(prev, b, ((at - r0) * c, 0.0, (at - r0) * s), ((at - r) * c, 0.0, (at - r) * s))
            prev, r0 = b, r
    return sc


SCENES = {"chain_64": lambda h: _chain(64, h), "chain_65": lambda h: _chain(65, h), "chain_69": lambda h: _chain(69, h),
          "chain_100": lambda h: _chain(100, h), "plate_30": lambda h: _chain(30, h, plate=True),
          "plate_40": lambda h: _chain(40, h, plate=True), "hub_6": lambda h: _hub(6, h), "hub_20": lambda h: _hub(20, h)}


# (a plate's chain at the first step only: the bounds are those of hanging chains,
# whose velocities are far above a resting contact's FP32 noise)
@pytest.mark.parametrize("name,k", [(n, k) for n in SCENES for k in (0, 12) if k == 0 or "plate" not in n])
@pytest.mark.parametrize("heavy", [True, False], ids=["fp64", "fp32"])
def test_single_step_parity_past_the_limits(name, heavy, k):
    import oracle
    sc = SCENES[name](heavy)
    g, p = cg.world(), oracle.port_world()
    for w in (g, p):
        scenes.apply(sc, w)
    if k > 0:
        g.step(k)
        p.set_state(**g.state())
        p.set_contacts(g.contacts())
        p.set_joint_state(g.joint_state())
    g.step(1)
    p.step(1)
    sg, sp = g.state(), p.state()
    dv = np.linalg.norm(sg["vel"] - sp["vel"], axis=1)
    vm = np.linalg.norm(sp["vel"], axis=1)
    dx = np.abs(sg["com"] - sp["com"]).max()
    stats = f"dv max {dv.max():.2e} median {np.median(dv):.2e} dx {dx:.2e}"
    assert np.all(dv <= 2e-3 + 2e-3 * vm), stats   # m/s
    assert dx <= 1e-4, stats                        # m
    jg, jp = g.joint_state()["impulse"], p.joint_state()["impulse"]
    assert np.abs(jg - jp).max() <= 1e-2 * (np.abs(jp).max() + 1.0), stats


@pytest.mark.parametrize("make", [lambda: _chain(33, True), lambda: _chain(60, False), lambda: _chain(34, True, plate=True),
                                  lambda: _chain(60, False, plate=True), lambda: _hub(20, True)],
                         ids=["chain_33", "chain_60", "plate_34", "plate_60", "hub_20"])
def test_held_islands_equal_those_in_global_memory(monkeypatch, make):
    out = []
    for cap in ("1536", "32"):   # islands of more than 32 bodies: held in shared memory, or not
        monkeypatch.setenv("CPGPU_PGS_DV_CAP", cap)
        w = cg.world()
        scenes.apply(make(), w)
        b = cg.Batch([w])
        st = []
        for _ in range(25):
            b.step(1)
            st.append(b.read_state().copy())
        out.append(np.stack(st).view(np.uint32))
    assert (out[0] == out[1]).all()
