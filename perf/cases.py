"""Performance cases: the calls a program makes into this framework, at the sizes it makes them.

Every case is a plain dict; `prepare` builds what a program holds before the
call (worlds, batches, ray and box arrays), `run` is one call as the program
makes it, and `listed` / `draw` give the sizes.  Kinds:

  world   one World stepped as an interactive program does: step(steps), then
          the bodies' state is read
  batch   a Batch of independent worlds stepped as a rollout loop does: the
          state is written from pinned host memory, stepped, and read back
  rays    World.raycast: host ray arrays against one world's bodies
  pairs   cpgpu_pairs_noalloc: candidate pairs of device AABBs into the
          caller's own device buffers
  serve   a Server: requests (clones of template worlds, each with a step
          count) submitted together and advanced until all are done

Scenes (the settings of each are those of constraintphysics_gb300.scenes):

  pile      random convex hulls of 8-32 points dropped on a plate
  pyramid   box pyramids
  drops     a mix of piles and pyramids
  mixed     boxes, spheres, cylinders, capsules and hulls on a plate (in a
            world of its own also bodies of several primitives)
  terrain   boxes, spheres and hulls on a triangle-mesh heightfield
  chains    articulated chains (ball-socket and hinge joints, block solve)
            swinging through fixed spheres, 8 substeps
  sleepers  stacks that fall asleep beside chains that keep swinging
"""
import ctypes
import functools
import math

import numpy as np
import torch

import constraintphysics_gb300 as cg
from constraintphysics_gb300 import scenes

M = scenes.PILE_MATERIAL


# ---------------------------------------------------------------- the cases ----
def listed():
    return [
        # the smallest interactive call: a dozen boxes, one step a frame
        {"name": "world_pyramid_14", "kind": "world", "scene": "pyramid", "bodies": 14, "steps": 1, "settle": 60},
        # the plain single-world path: 1,000 hulls in one pile
        {"name": "world_pile_1000", "kind": "world", "scene": "pile", "bodies": 1000, "steps": 1, "settle": 240},
        # an interactive scene with sleeping enabled, most of it at rest
        {"name": "world_sleepers_2400", "kind": "world", "scene": "sleepers", "bodies": 2400, "steps": 1, "settle": 90},
        # one large world on a triangle mesh
        {"name": "terrain_20000", "kind": "batch", "scene": "terrain", "bodies": 20000, "worlds": 1, "low": 20000,
         "steps": 1, "settle": 120},
        # the batched workload: 4,096 worlds of 8-512 bodies, every step through host memory
        {"name": "batch_drops_4096", "kind": "batch", "scene": "drops", "worlds": 4096, "low": 8, "bodies": 512,
         "steps": 1, "settle": 60},
        # a small batch of small worlds, a few steps a call (frame skip)
        {"name": "batch_drops_60", "kind": "batch", "scene": "drops", "worlds": 60, "low": 8, "bodies": 64, "steps": 4,
         "settle": 90},
        # every kind of shape
        {"name": "batch_mixed_333", "kind": "batch", "scene": "mixed", "worlds": 333, "low": 9, "bodies": 100, "steps": 2,
         "settle": 90},
        # articulated chains: joints, 8 substeps, the holonomic block solve
        {"name": "batch_chains_512", "kind": "batch", "scene": "chains", "worlds": 512, "low": 16, "bodies": 64,
         "steps": 1, "settle": 30},
        # a sensor's fan of rays into a scene
        {"name": "rays_4096", "kind": "rays", "bodies": 1000, "rays": 4096},
        # the broadphase alone, at its largest and at an ordinary size
        {"name": "pairs_65536", "kind": "pairs", "bodies": 65536, "order": "random"},
        {"name": "pairs_1021", "kind": "pairs", "bodies": 1021, "order": "random"},
        # requests of mixed sizes served together
        {"name": "serve_96", "kind": "serve", "requests": 96, "low": 16, "bodies": 256, "max_steps": 40},
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    kind = rng.choice(["world", "world", "batch", "batch", "batch", "rays", "pairs", "serve"])
    if kind == "world":
        scene = rng.choice(["pyramid", "pile", "mixed", "sleepers"])
        n = _log(rng, 8, 1000) if scene != "sleepers" else _log(rng, 100, 2400)
        return {"kind": kind, "scene": scene, "bodies": n, "steps": rng.choice([1, 1, 2, 5]), "settle": 90}
    if kind == "batch":
        scene = rng.choice(["drops", "drops", "mixed", "chains", "terrain"])
        if scene == "terrain":
            worlds, n = 1, _log(rng, 200, 20000)
            return {"kind": kind, "scene": scene, "bodies": n, "worlds": worlds, "low": n, "steps": rng.choice([1, 2]),
                    "settle": 120}
        low = 8 if scene != "chains" else 16
        top = {"drops": 512, "mixed": 100, "chains": 64}[scene]
        n = _log(rng, low + 4, top)
        worlds = _log(rng, 2, {"drops": 1500, "mixed": 300, "chains": 300}[scene])
        return {"kind": kind, "scene": scene, "worlds": worlds, "low": low, "bodies": n, "steps": rng.choice([1, 2, 4]),
                "settle": 60 if scene != "chains" else 30}
    if kind == "rays":
        return {"kind": kind, "bodies": _log(rng, 10, 2000), "rays": _log(rng, 1, 16384)}
    if kind == "pairs":
        return {"kind": kind, "bodies": _log(rng, 16, 65536), "order": rng.choice(["random", "grid"])}
    return {"kind": kind, "requests": _log(rng, 4, 96), "low": 16, "bodies": _log(rng, 24, 256), "max_steps": 40}


# ---------------------------------------------------------------- scenes ----
@functools.lru_cache(maxsize=1)
def _pool():
    """Unit hull shapes reused by every scene (the scenes scale, place and turn them)."""
    return scenes.HullPool(0, size=256)


def _drop(rng, n, kind=None):
    """A pile or a pyramid of n bodies (either, where kind is None)."""
    while True:
        sc = scenes.batched_world(rng, _pool(), n + 0.5, n + 0.5)
        if kind is None or sc.name.startswith(kind):
            return sc


def _body(sc, rng, pos, round_ends=False, unions=False):
    u = rng.random()
    if u < 0.35:
        d = rng.uniform(0.5, 1.5, size=3)
        bid = sc.box((-d[0] / 2, -d[1] / 2, -d[2] / 2), d[0], d[1], d[2], M, scenes.DYNAMIC, pos)
    elif u < 0.55:
        bid = sc.sphere((0.0, 0.0, 0.0), rng.uniform(0.3, 0.8), M, scenes.DYNAMIC, pos)
    elif u < 0.7 and round_ends:
        r, h = rng.uniform(0.3, 0.6), rng.uniform(0.5, 1.5)
        bid = sc.cylinder((0.0, -h / 2, 0.0), r, h, M, scenes.DYNAMIC, pos)
    elif u < 0.8 and round_ends:
        r, h = rng.uniform(0.25, 0.5), rng.uniform(0.3, 1.2)
        bid = sc.capsule((0.0, -h / 2, 0.0), r, h, M, scenes.DYNAMIC, pos)
    elif u < 0.87 and unions:
        prims = [("capsule", (0.0, -0.6, 0.0), 0.15, 1.2, M), ("sphere", (0.0, 0.75, 0.0), 0.35, M),
                 ("sphere", (0.0, -0.75, 0.0), 0.35, M)]
        bid = sc.union(prims, scenes.DYNAMIC, pos)
    else:
        pts, faces = _pool().draw(rng)
        bid = sc.hull(pts, faces, M, scenes.DYNAMIC, pos)
    sc.orient(bid, scenes.random_quat(rng))


def _mixed(rng, n, unions):
    sc = scenes.Scene("mixed_%d" % n, scenes.MIXED_PARAMS)
    sc.box((-250.0, -2.0, -250.0), 500.0, 2.0, 500.0, M, scenes.FIXED)
    side = max(1, int(math.ceil((n / 3.0) ** 0.5)))
    off = (side - 1) * 1.6
    for k in range(n):
        j, i = divmod(k, side * side)
        pos = np.array([(i % side) * 3.2 - off, 2.0 + 3.2 * j, (i // side) * 3.2 - off]) + rng.uniform(-0.1, 0.1, size=3)
        _body(sc, rng, pos, True, unions)
    return sc


@functools.lru_cache(maxsize=4)
def _ground(grid):
    """A heightfield of grid x grid metres: heights, points, triangles."""
    h = scenes.value_noise(np.random.default_rng(grid), grid)
    pts, tris = scenes.grid_mesh(h, 1.0, (-grid / 2.0, 0.0, -grid / 2.0))
    return h, pts, tris


def _terrain(rng, n):
    """n mixed bodies in four layers above the ground under them (71 x 71 a layer at 20,000)."""
    side = max(4, int(math.ceil((n / 4.0) ** 0.5)))
    grid = 16
    while grid < 3.2 * side + 8:
        grid *= 2
    h, pts, tris = _ground(grid)
    sc = scenes.Scene("terrain_%d" % n, scenes.MIXED_PARAMS)
    sc.mesh(pts, tris, M)
    off = (side - 1) * 1.6
    for k in range(n):
        j, i = divmod(k, side * side)
        x, z = (i % side) * 3.2 - off, (i // side) * 3.2 - off
        y = float(h[int(x + grid / 2), int(z + grid / 2)])
        _body(sc, rng, np.array([x, y + 2.5 + 3.2 * j, z]) + rng.uniform(-0.1, 0.1, size=3))
    return sc


def _world(sc):
    w = cg.world()
    scenes.apply(sc, w)
    return w


def _scene(case, rng, n):
    kind = case["scene"]
    if kind == "mixed":
        return _mixed(rng, n, case["kind"] == "world")
    if kind == "terrain":
        return _terrain(rng, n)
    if kind == "chains":
        return scenes.chain_world(rng, n, n)
    if kind == "sleepers":
        # about n bodies: stacks of three with a ball at every third, and a hung chain of eight for each 15 stacks
        stacks = max(3, int(n / 3.94))
        return scenes.large_mixed_world(int(rng.integers(1 << 30)), stacks, max(1, stacks // 15))
    return _drop(rng, n, None if kind == "drops" else kind)


def _sizes(case, count):
    """Log-uniform body counts, the same for every seed (so is the outputs' shape)."""
    rng = np.random.default_rng(count)
    lo, hi = math.log(case["low"]), math.log(case["bodies"] + 1)
    return [min(case["bodies"], int(math.exp(rng.uniform(lo, hi)))) for _ in range(count)]


# ---------------------------------------------------------------- rays ----
def _ray_scene(case, seed):
    """Boxes, spheres and cylinders at random poses in a room, and rays from its middle outwards."""
    rng = np.random.default_rng(seed)
    n, m = case["bodies"], case["rays"]
    half = 2.2 * n ** (1.0 / 3.0) + 3.0
    kind = rng.integers(0, 3, size=n)
    size = np.where(kind[:, None] == 0, rng.uniform(0.5, 1.5, size=(n, 3)), rng.uniform(0.3, 0.8, size=(n, 3)))
    pos = rng.uniform(-half, half, size=(n, 3))
    pos[np.linalg.norm(pos, axis=1) < 3.0] += 4.0
    quat = rng.normal(size=(n, 4))
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    org = rng.uniform(-1.0, 1.0, size=(m, 3))
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return kind, size, pos, quat, org, d


def _rot(q):
    r, i, j, k = q
    return np.array([[r * r + i * i - j * j - k * k, 2 * i * j - 2 * r * k, 2 * i * k + 2 * r * j],
                     [2 * i * j + 2 * r * k, r * r - i * i + j * j - k * k, 2 * j * k - 2 * r * i],
                     [2 * i * k - 2 * r * j, 2 * j * k + 2 * r * i, r * r - i * i - j * j + k * k]])


def _exact_rays(case, seed):
    """The first hit of every ray in 64 bits, from the shapes' own equations (a
    cap's normal is the cylinder's axis on both ends, as the engine defines it)."""
    kind, size, pos, quat, org, d = _ray_scene(case, seed)
    m = len(org)
    best = np.full(m, np.inf)
    nrm = np.zeros((m, 3))
    for b in range(len(kind)):
        R = _rot(quat[b])
        o, v = (org - pos[b]) @ R, d @ R          # in the body's frame
        with np.errstate(divide="ignore", invalid="ignore"):
            if kind[b] == 1:
                B, C = (o * v).sum(1), (o * o).sum(1) - size[b, 0] ** 2
                q = B * B - C
                t = np.where(q >= 0, -B - np.sqrt(np.maximum(q, 0)), np.inf)
                n = o + t[:, None] * v
            else:
                if kind[b] == 0:
                    h = size[b] / 2
                    near = np.minimum((-h - o) / v, (h - o) / v)
                    far = np.maximum((-h - o) / v, (h - o) / v)
                    ax = near.argmax(1)
                    t0, t1 = near.max(1), far.min(1)
                    n = np.zeros((m, 3))
                    n[np.arange(m), ax] = -np.sign(v[np.arange(m), ax])
                else:
                    r, h = size[b, 0], size[b, 1] / 2
                    a = v[:, 0] ** 2 + v[:, 2] ** 2
                    B, C = o[:, 0] * v[:, 0] + o[:, 2] * v[:, 2], o[:, 0] ** 2 + o[:, 2] ** 2 - r * r
                    q = B * B - a * C
                    s = np.sqrt(np.maximum(q, 0))
                    side0, side1 = np.where(q >= 0, (-B - s) / a, np.inf), np.where(q >= 0, (-B + s) / a, -np.inf)
                    c0, c1 = np.minimum((-h - o[:, 1]) / v[:, 1], (h - o[:, 1]) / v[:, 1]), \
                        np.maximum((-h - o[:, 1]) / v[:, 1], (h - o[:, 1]) / v[:, 1])
                    t0, t1 = np.maximum(side0, c0), np.minimum(side1, c1)
                    p = o + t0[:, None] * v
                    n = np.where((c0 > side0)[:, None], np.array([0.0, 1.0, 0.0]),
                                 np.stack([p[:, 0], 0 * t0, p[:, 2]], 1))
                t = np.where(t0 <= t1, t0, np.inf)
        hit = (t > 0) & (t < best)
        best[hit] = t[hit]
        nrm[hit] = (n[hit] / np.linalg.norm(n[hit], axis=1, keepdims=True)) @ R.T
    miss = ~np.isfinite(best)
    p = org + np.where(miss, 0.0, best)[:, None] * d
    p[miss] = 0.0
    return {"body": None, "pos": p, "normal": nrm, "dist": np.where(miss, -1.0, best)}


# ---------------------------------------------------------------- the entry points ----
@functools.lru_cache(maxsize=1)
def _pairs_fn():
    fn = cg.lib()._lib.cpgpu_pairs_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    return fn


def _boxes(case, seed):
    """Body-sized AABBs, about three overlaps a body, in creation order along a grid or in no order."""
    rng = np.random.default_rng(seed)
    n = case["bodies"]
    side = int(math.ceil(n ** (1.0 / 3.0)))
    k = np.arange(side ** 3)
    cells = np.stack([k % side, k // side % side, k // (side * side)], 1)[:n].astype(np.float64)
    c = cells * 1.1 + rng.uniform(-0.5, 0.5, size=(n, 3))
    if case["order"] == "random":
        c = c[rng.permutation(n)]
    h = rng.uniform(0.3, 0.75, size=(n, 3))
    return np.concatenate([c - h, c + h], 1).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind}
    if kind == "world":
        w = _world(_scene(case, rng, case["bodies"]))
        w.step(case["settle"])
        s.update(world=w, steps=case["steps"])
    elif kind == "batch":
        # up to 64 different worlds, repeated; the repetitions part from each
        # other by the velocities written below
        n = case["worlds"]
        own = [_world(_scene(case, rng, b)) for b in _sizes(case, min(n, 64))]
        worlds = own + [cg.clone(own[i % len(own)]) for i in range(len(own), n)]
        b = cg.Batch(worlds)
        host = torch.empty((b.n_bodies, 16), dtype=torch.float32, pin_memory=True)
        b.read_state(host)
        g = torch.Generator().manual_seed(int(seed))
        host[:, 8:11] += 0.05 * torch.randn((b.n_bodies, 3), generator=g)
        b.write_state(host)
        b.step(case["settle"])
        b.read_state(host)
        s.update(batch=b, host=host, out=torch.empty_like(host).pin_memory(), steps=case["steps"])
    elif kind == "rays":
        shapes, size, pos, quat, org, d = _ray_scene(case, seed)
        w = cg.world()
        w.set_params(**scenes.MIXED_PARAMS)
        for k in range(len(shapes)):
            if shapes[k] == 0:
                x, y, z = size[k]
                bid = w.add_box((-x / 2, -y / 2, -z / 2), x, y, z, M, scenes.DYNAMIC, pos[k])
            elif shapes[k] == 1:
                bid = w.add_sphere((0.0, 0.0, 0.0), size[k, 0], M, scenes.DYNAMIC, pos[k])
            else:
                bid = w.add_cylinder((0.0, -size[k, 1] / 2, 0.0), size[k, 0], size[k, 1], M, scenes.DYNAMIC, pos[k])
            w.set_orientation(bid, quat[k])
        w.aabbs()   # the world is on the device before the first query
        s.update(world=w, org=org, dirs=d)
    elif kind == "pairs":
        n = case["bodies"]
        cap = 16 * n
        s.update(boxes=torch.from_numpy(_boxes(case, seed)).cuda(), n=n, cap=cap,
                 pairs=torch.zeros((cap, 2), dtype=torch.int32, device="cuda"),
                 count=torch.zeros(1, dtype=torch.int32, device="cuda"))
    else:
        own = [_world(_drop(rng, b)) for b in _sizes(case, min(case["requests"], 24))]
        steps = [int(rng.integers(case["max_steps"] // 4, case["max_steps"] + 1)) for _ in range(case["requests"])]
        s.update(templates=own, steps=steps, server=cg.Server(32 << 30, 10))
    return s


def run(s):
    kind = s["kind"]
    if kind == "world":
        s["world"].step(s["steps"])
        return s["world"].state()
    if kind == "batch":
        b = s["batch"]
        b.write_state(s["host"])
        b.step(s["steps"])
        b.read_state(s["out"])
        return s["out"]
    if kind == "rays":
        return s["world"].raycast(s["org"], s["dirs"])
    if kind == "pairs":
        rc = _pairs_fn()(s["boxes"].data_ptr(), s["n"], s["pairs"].data_ptr(), s["cap"], s["count"].data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("cpgpu_pairs_noalloc: status %d" % rc)
        return s["pairs"], s["count"]
    srv, got = s["server"], {}
    for i, k in enumerate(s["steps"]):
        w = cg.clone(s["templates"][i % len(s["templates"])])
        got[srv.submit(w, k)] = (i, w)
    worlds = [None] * len(got)
    while got:
        srv.advance(10)
        for tok in srv.poll():
            i, w = got.pop(tok)
            worlds[i] = w
    st = [w.state() for w in worlds]
    return {k: np.concatenate([x[k] for x in st]) for k in ("com", "quat", "vel", "ang_vel")}


# ---------------------------------------------------------------- its work ----
# Per body of a settled scene: candidate pairs, contact points, and the passes
# over the contacts of one substep.
_PER_BODY = {"pile": (2.5, 5.0, 11), "pyramid": (1.5, 6.0, 11), "drops": (1.5, 5.3, 11), "mixed": (2.0, 3.0, 21),
             "terrain": (2.0, 3.0, 21), "chains": (0.5, 0.1, 5), "sleepers": (1.0, 1.0, 11)}


def _step_work(scene, bodies, steps):
    """Bytes: the bodies' state (pose, velocities, inertia) and the contacts'
    stored state read and written once a step, the shapes read once.  Flops:
    the axis tests of a pair, and a contact's three rows (three 12-term dot
    products and updates) in every pass; joints as 4 rows of 12 terms in 6
    passes of 8 substeps."""
    pairs, contacts, passes = _PER_BODY[scene]
    nbytes = 2 * 168 + 2 * 140 * contacts + 8 * pairs + 600
    flops = 4000 * pairs + contacts * (600 + 160 * passes) + 500
    if scene == "chains":
        nbytes, flops = nbytes + 8 * 300, flops + 8 * 6 * 4 * 48 + 8 * 1000
    return {"bytes": nbytes * bodies * steps, "flops": flops * bodies * steps}


def work(case):
    kind = case["kind"]
    if kind == "world":
        w = _step_work(case["scene"], case["bodies"], case["steps"])
        return {"bytes": w["bytes"] + 52 * case["bodies"], "flops": w["flops"]}
    if kind in ("batch", "serve"):
        lo, hi = float(case["low"]), float(case["bodies"] + 1)
        mean = (hi - lo) / math.log(hi / lo) if hi > lo + 1 else lo     # of a log-uniform size
        if kind == "serve":
            n = mean * case["requests"]
            w = _step_work("drops", n, 0.625 * case["max_steps"])
            return {"bytes": w["bytes"] + 52 * n, "flops": w["flops"]}
        n = mean * case["worlds"]
        w = _step_work(case["scene"], n, case["steps"])
        return {"bytes": w["bytes"] + 2 * 64 * n, "flops": w["flops"]}
    if kind == "rays":
        return {"bytes": 100 * case["bodies"] + (24 + 32) * case["rays"], "flops": 30.0 * case["rays"] * case["bodies"] ** (1 / 3.0)}
    return {"bytes": (24 + 8 * 3) * case["bodies"], "flops": 6.0 * 27 * case["bodies"]}


def exact(case, seed):
    """Ray hits have exact values; a step of contacts is one of many valid
    roundings of a discontinuous map, and pairs are whole numbers."""
    return _exact_rays(case, seed) if case["kind"] == "rays" else None
