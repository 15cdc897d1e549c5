"""Performance cases of the rigid-body step: what a program that uses this framework has it do.

Every case goes through the package's public entry points (``GpuWorld``, ``Server``).  Most are the
call of a simulation loop that owns the state between calls (a game loop, a batch of training
environments, a planner's rollouts): the poses and velocities go in from page-locked host arrays in
the world's real type, the world advances by one or a few steps, and the new poses and velocities
come back.  The worlds have settled first, so that the contacts, islands and contact pools are those
of a running simulation.  Sizes are those of this repository's benchmark configurations, tests and
demos.

Families (``"family"`` of a case):
  pile     one world of mixed boxes, spheres, cylinders and convex hulls on a ground box
  tower    boxes stacked with 1 mm gaps and hit by a sphere, contact margin 5 mm, 20 iterations
  cube     mixed primitives scattered in a cube: many pairs, few contacts (no settling)
  pour     bodies poured into a walled container: one large scene, islands of many contacts
  batch    many independent piles of uneven size in one world (batched environments)
  chains   jointed chains (ball joints, limited and motor hinges, sliders) over a ground box
  terrain  bodies of every kind, compounds among them, on a concave heightfield
  burst    requests of different sizes and step counts served by the request loop until all are done
  solve    contacts from the caller's own collision detection, solved for the new velocities
"""
import math
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parent.parent / "physics-engine_gb300"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import pe_gb300 as pg  # noqa: E402
from pe_gb300 import scene as sc  # noqa: E402

FIELDS = ("origin", "basis", "lin_vel", "ang_vel")
SHAPES = {"origin": (3,), "basis": (3, 3), "lin_vel": (3,), "ang_vel": (3,)}
MODES = {"serial": pg.SERIAL_ORDER, "coloured": pg.COLORED}


def case(family, name=None, **kw):
    c = {"family": family, "bits": 32, "mode": "coloured", "steps": 1, **kw}
    return {**c, "name": name} if name else c


def listed():
    return [
        # the smallest scene that a program steps: a handful of bodies, one step per frame
        case("pile", "pile_12", n=12, settle=90),
        # an ordinary scene of a game or an editor, an odd body count, hulls of up to 64 vertices
        case("pile", "pile_501", n=501, settle=120),
        # the stacked tower at the sphere's impact, one island, in single precision
        case("tower", "tower_1000_f32", nx=10, ny=10, nz=10, settle=30),
        # the same in the reference's default precision and its exact constraint order
        case("tower", "tower_1000_f64_serial", nx=10, ny=10, nz=10, settle=30, bits=64, mode="serial"),
        # pair-finding and closed-form contacts: 65,536 scattered bodies
        case("cube", "cube_65536", n=65536, extent=100.0),
        # one large scene: bodies poured into a container, thousands of contacts per island
        case("pour", "pour_40000", n=40000, settle=180),
        # a planner's or trainer's small batch, four steps per call (action repeat)
        case("batch", "batch_48_rollout4", scenes=48, settle=120, steps=4),
        # the batched configuration: 4,096 uneven piles, about half a million bodies
        case("batch", "batch_4096", scenes=4096, settle=120),
        # machinery: jointed chains with limits and motors, double precision, exact order
        case("chains", "chains_200_f64_serial", chains=200, links=7, settle=60, bits=64, mode="serial"),
        # a level: compounds, hulls and primitives on a triangle-mesh terrain
        case("terrain", "terrain_300", n=300, cells=48, settle=60),
        # serving: requests of 16 to 256 bodies and 4 to 24 steps, admitted and retired as they go
        case("burst", "burst_16", requests=16, most=256),
        # the solver behind the caller's own narrowphase
        case("solve", "solve_6000", n=6000),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(("pile", "pile", "tower", "cube", "pour", "batch", "batch", "chains", "terrain", "burst", "solve"))
    bits = rng.choice((32, 32, 32, 64))
    mode = rng.choice(("coloured", "coloured", "serial"))
    opt = dict(bits=bits, mode=mode, steps=rng.choice((1, 1, 1, 2, 4)))
    if family == "pile":
        return case(family, n=spread(8, 700 if bits == 32 else 300), settle=rng.randrange(60, 140), **opt)
    if family == "tower":
        top = 10 if bits == 32 else 8
        return case(family, nx=rng.randint(2, top), ny=rng.randint(3, top), nz=rng.randint(2, top),
                    settle=rng.randrange(20, 50), **dict(opt, steps=1))
    if family == "cube":
        n = spread(1000, 65536 if bits == 32 else 30000)
        return case(family, n=n, extent=round(100.0 * (n / 65536.0) ** (1 / 3) * rng.uniform(0.9, 1.2), 3), **dict(opt, steps=1))
    if family == "pour":   # coloured: how a scene this size is run
        return case(family, n=spread(2000, 40000), settle=rng.randrange(120, 200), **dict(opt, bits=32, mode="coloured", steps=1))
    if family == "batch":
        return case(family, scenes=spread(4, 2000 if bits == 32 else 60), settle=rng.randrange(90, 130), **opt)
    if family == "chains":
        return case(family, chains=spread(4, 300), links=rng.randint(3, 9), settle=rng.randrange(30, 70), **opt)
    if family == "terrain":
        return case(family, n=spread(20, 400), cells=rng.randint(12, 56), settle=rng.randrange(40, 70), **opt)
    if family == "burst":
        return case(family, requests=spread(4, 24), most=spread(32, 300), **dict(opt, bits=32, steps=1))
    return case(family, n=spread(30, 20000 if bits == 32 else 6000), **dict(opt, steps=1))


# ------------------------------------------------------------------ inputs
def _scene(c, seed):
    """(Scene, scene offsets or None) of a case."""
    f, bits = c["family"], c["bits"]
    if f == "pile":
        return sc.pile(c["n"], seed=seed, drop=(0.0, 1.0), real_bits=bits), None
    if f == "tower":   # the sphere's speed and the tower's friction vary with the seed
        r = np.random.default_rng(seed)
        return sc.tower(c["nx"], c["ny"], c["nz"], sphere_speed=30.0 + r.uniform(-2, 2), friction=r.uniform(0.45, 0.55),
                        real_bits=bits), None
    if f == "cube":
        return _cube(c["n"], c["extent"], seed, bits), None
    if f == "pour":
        side = (c["n"] / 4.1) ** (1 / 3)   # the density of 262,144 bodies in 40 x 40 x 80 m
        return sc.container_pour(c["n"], seed=seed, floor=(side, side), spawn_height=(0.5, 0.5 + 2 * side),
                                 wall_height=2 * side + 10, real_bits=bits), None
    if f == "batch":   # the environments are the case's, their starts the seed's
        s, offs = _environments(c["scenes"], bits)
        r = np.random.default_rng(seed)
        n, moves = s.n_bodies, (s.body_flags == 0)
        v = np.where(moves[:, None], r.normal(0, 0.5, (n, 3)), 0.0)
        basis = np.where(moves[:, None, None], sc.random_rotations(r, n), s.basis)
        s = sc.dataclasses.replace(s, lin_vel=v, basis=basis)
        return (s.rounded(bits) if bits == 32 else s), offs
    if f == "chains":
        return sc.chain_field(c["chains"], c["links"], seed=seed, real_bits=bits), None
    return sc.terrain_drop(c["n"], c["cells"], c["cells"], seed=seed, real_bits=bits), None


def _cube(n, extent, seed, bits):
    """Boxes, spheres and cylinders (60/25/15) of 0.2 to 1 m at random places in a cube, with random
    rotations and velocities: ``scene.random_cube`` laid out as arrays."""
    r = np.random.default_rng(seed)
    s = sc.Scene(dt=1.0 / 60.0, iterations=10)
    kind = r.choice(3, size=n, p=(0.60, 0.25, 0.15)).astype(np.int32)
    he, rs, rc, hc = r.uniform(0.2, 1.0, (n, 3)), r.uniform(0.2, 1.0, n), r.uniform(0.2, 0.8, n), r.uniform(0.4, 2.0, n)
    par = np.where((kind == sc.BOX)[:, None], 2 * he, 0.0)
    par[kind == sc.SPHERE, 0] = rs[kind == sc.SPHERE]
    par[kind == sc.CYLINDER, 0], par[kind == sc.CYLINDER, 1] = rc[kind == sc.CYLINDER], hc[kind == sc.CYLINDER]
    vol = np.where(kind == sc.BOX, np.prod(2 * he, axis=1), np.where(kind == sc.SPHERE, 4 / 3 * np.pi * rs ** 3, np.pi * rc * rc * hc))
    s.shape_type, s.shape_param = kind, par
    s.hull_vbeg = s.hull_vcnt = s.hull_fbeg = s.hull_fcnt = np.zeros(n, np.int32)
    s.hull_verts, s.hull_face_off, s.hull_face_idx = np.zeros((0, 3)), np.zeros(1, np.int32), np.zeros(0, np.int32)
    _bodies(s, np.arange(n, dtype=np.int32), np.zeros(n, np.int32), 1000.0 * vol, r.uniform(0, extent, (n, 3)),
            sc.random_rotations(r, n), r.normal(0, 2.0, (n, 3)), np.zeros((n, 3)))
    return s.rounded(bits) if bits == 32 else s


def _bodies(s, shape, flags, mass, origin, basis, v, w):
    n = len(shape)
    s.body_shape, s.body_flags, s.mass = shape, flags, mass
    s.friction, s.restitution = np.full(n, 0.5), np.zeros(n)
    s.lin_damp, s.ang_damp = np.zeros(n), np.zeros(n)
    s.origin, s.basis, s.lin_vel, s.ang_vel = origin, basis, v, w


def _pinned(a):
    """The array's copy in page-locked memory, as a loop that transfers every step keeps it."""
    t = torch.from_numpy(np.ascontiguousarray(a))
    if torch.cuda.is_available():
        t = t.pin_memory()
    return t.numpy()


def _buffers(n, dtype, fields=FIELDS):
    return {k: _pinned(np.zeros((n,) + SHAPES[k], dtype)) for k in fields}


@lru_cache(maxsize=2)
def _environments(n, bits):
    """``n`` piles of 8 to 512 bodies (log-uniform) with hulls from a shared pool of shapes."""
    return sc.batched_piles(n, seed=4096 + n, drop=(0.0, 5.0), hull_pool=min(512, 16 + n), real_bits=bits)


@lru_cache(maxsize=4)
def _catalogue(most):
    """The scenes that a service's clients ask for: piles of 16 to ``most`` bodies."""
    sizes = np.unique(np.geomspace(16, most, 12).astype(int))
    return [sc.pile(int(n), seed=97 + int(n), drop=(0.0, 0.5), real_bits=32) for n in sizes]


def prepare(c, seed):
    family = c["family"]
    if family == "solve":
        return _prepare_solve(c, seed)
    if family == "burst":
        pool, asked = _catalogue(c["most"]), np.random.default_rng(c["requests"])   # what is asked for
        r = np.random.default_rng(seed)                                             # and from which start
        asks = []
        for _ in range(c["requests"]):
            s = pool[int(asked.integers(len(pool)))]
            v = r.uniform(-1, 1, s.lin_vel.shape).astype(np.float32) * (s.body_flags == 0)[:, None]
            asks.append((sc.dataclasses.replace(s, lin_vel=v.astype(np.float64)), int(asked.integers(4, 25))))
        return dict(family=family, server=pg.Server(real_bits=32, mode=MODES[c["mode"]]), asks=asks)
    s, offs = _scene(c, seed)
    margin = 0.005 if family == "tower" else 0.0
    world = pg.GpuWorld(s, c["bits"], scenes=offs, margin=margin, tuning="auto")
    mode = MODES[c["mode"]]
    if c.get("settle"):   # the settling steps run in the order that a program of this size uses
        world.step(c["settle"], mode)
    dtype = np.float32 if c["bits"] == 32 else np.float64
    now = world.state(FIELDS, dtype=dtype)
    return dict(family=family, world=world, mode=mode, steps=c["steps"], dt=s.dt, moves=np.asarray(s.body_flags) == 0,
                inputs={k: _pinned(now[k]) for k in FIELDS}, out=_buffers(s.n_bodies, dtype))


# ------------------------------------------------------------------ one pass
def run(state):
    family = state["family"]
    if family == "burst":
        server = state["server"]
        ids = [server.submit(s, k) for s, k in state["asks"]]
        live = queued = 1
        while live or queued:
            live, queued = server.step()
        done = [server.result(i)[1] for i in ids]
        return {k: np.concatenate([d[k] for d in done]).astype(np.float32) for k in FIELDS}
    world = state["world"]
    world.set_state(state["inputs"])
    if family == "solve":
        world.solve(state["mode"])
        return world.state(out=state["out"], fields=("lin_vel", "ang_vel"))
    world.step(state["steps"], state["mode"])
    out = dict(world.state(FIELDS, out=state["out"]))
    n = world.last_counts()
    out["counts"] = np.array([n["pairs"], n["active"], n["rows"], n["islands"]], np.int32)
    return out


# ------------------------------------------------------------------ the least that a pass can do
def work(c):
    """Bytes: each body's pose, velocities and constants read once, poses and velocities written once,
    and the shapes' data once.  Flops: about 250 for a body's integration and bounds, 60 for a pair's
    test, and 160 for each contact point and solver iteration, with typical counts of each per body."""
    real = c["bits"] // 8
    pairs, points, iters = 3.0, 2.5, 10
    hulls = 0.0
    family = c["family"]
    if family == "tower":
        bodies, pairs, points, iters = c["nx"] * c["ny"] * c["nz"] + 2, 5.0, 5.0, 20
    elif family == "batch":
        bodies, hulls = c["scenes"] * 122, 0.2
    elif family == "chains":
        bodies, points = c["chains"] * (c["links"] + 1) + 1, 1.5
    elif family == "burst":
        bodies, hulls = c["requests"] * (c["most"] - 16) / max(math.log(c["most"] / 16.0), 1e-3), 0.2
    elif family == "cube":
        bodies, pairs, points = c["n"], 1.2, 1.1
    elif family == "solve":
        bodies, pairs, points = c["n"], 0.0, 4.0
        return {"bytes": bodies * real * (12 + 6 + 10 + 6) + bodies * points * real * 19, "flops": bodies * points * iters * 160.0}
    else:
        bodies, hulls = c["n"] + 1, 0.2
    steps = c["steps"] if family != "burst" else 14
    per_step = 250.0 + 60.0 * pairs + 160.0 * points * iters
    return {"bytes": bodies * real * (18 + 16 + 18 + 3 + hulls * 36 * 3), "flops": bodies * per_step * steps}


# ------------------------------------------------------------------ values in 64 bits
def exact(c, seed):
    """One step's poses follow from its inputs alone (velocities are applied before contacts are
    found); the solver's velocities follow from its contacts.  Velocities after a whole step, and
    whatever takes several steps, hang on contact decisions and have no value of their own."""
    if c["family"] == "solve":
        return _exact_solve(c, seed)
    if c["family"] == "burst" or c["steps"] != 1:
        return None
    state = prepare(c, seed)
    o, b, v, w = (np.asarray(state["inputs"][k], np.float64) for k in FIELDS)
    dt, moves = state["dt"], state["moves"]
    q = _quaternions(b)
    half = 0.5 * dt * w
    # q + (half, 0) * q, normalised
    x, y, z, s = q.T
    hx, hy, hz = half.T
    q2 = np.stack([x + hx * s + hy * z - hz * y, y + hy * s + hz * x - hx * z, z + hz * s + hx * y - hy * x,
                   s - hx * x - hy * y - hz * z], axis=1)
    q2 /= np.linalg.norm(q2, axis=1, keepdims=True)
    o2 = np.where(moves[:, None], o + v * dt, o)
    b2 = np.where(moves[:, None, None], sc.quat_to_basis(q2[:, [3, 0, 1, 2]]), b)
    state["world"].close()
    return {"origin": o2, "basis": b2, "lin_vel": None, "ang_vel": None, "counts": None}


def _quaternions(m):
    """(x, y, z, w) of rotation matrices, from the largest of the four components."""
    d = np.stack([1 + m[:, 0, 0] - m[:, 1, 1] - m[:, 2, 2], 1 - m[:, 0, 0] + m[:, 1, 1] - m[:, 2, 2],
                  1 - m[:, 0, 0] - m[:, 1, 1] + m[:, 2, 2], 1 + m[:, 0, 0] + m[:, 1, 1] + m[:, 2, 2]], axis=1)
    r = [m[:, 2, 1] - m[:, 1, 2], m[:, 0, 2] - m[:, 2, 0], m[:, 1, 0] - m[:, 0, 1]]
    p = [m[:, 0, 1] + m[:, 1, 0], m[:, 0, 2] + m[:, 2, 0], m[:, 1, 2] + m[:, 2, 1]]
    cand = np.stack([np.stack([d[:, 0], p[0], p[1], r[0]], 1), np.stack([p[0], d[:, 1], p[2], r[1]], 1),
                     np.stack([p[1], p[2], d[:, 2], r[2]], 1), np.stack([r[0], r[1], r[2], d[:, 3]], 1)], axis=1)
    q = cand[np.arange(len(m)), np.argmax(d, axis=1)]
    q = q / np.linalg.norm(q, axis=1, keepdims=True)
    return np.where(q[:, 3:] < 0, -q, q)


# ------------------------------------------------------------------ contacts of the caller's own
def _contacts(c, seed):
    """Boxes in columns on a floor, a few degrees off the upright, each column's neighbours touching
    at four points: the arrays of a caller's collision detection, in the world's precision."""
    real = np.float32 if c["bits"] == 32 else np.float64
    r = np.random.default_rng(seed)
    n = c["n"]
    high = int(min(12, max(2, round(n ** (1 / 3)))))
    cols = -(-n // high)
    wide = int(math.ceil(math.sqrt(cols)))
    level, col = np.arange(n) // cols, np.arange(n) % cols
    size = np.stack([r.uniform(0.8, 1.2, n), np.ones(n), r.uniform(0.8, 1.2, n)], axis=1).astype(real).astype(np.float64)
    origin = np.stack([(col % wide) * 1.1, 0.5 + 0.995 * level, (col // wide) * 1.1], axis=1) + r.uniform(-0.02, 0.02, (n, 3))
    angle = r.normal(0, 0.02, (n, 3))
    half = 0.5 * angle
    q = np.concatenate([half, np.ones((n, 1))], axis=1)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    basis = sc.quat_to_basis(q[:, [3, 0, 1, 2]])
    s = sc.Scene(dt=1.0 / 60.0, iterations=10)
    floor = np.array([wide * 1.1 + 20.0, 1.0, wide * 1.1 + 20.0])
    s.shape_type, s.shape_param = np.zeros(n + 1, np.int32), np.concatenate([floor[None], size])
    s.hull_vbeg = s.hull_vcnt = s.hull_fbeg = s.hull_fcnt = np.zeros(n + 1, np.int32)
    s.hull_verts, s.hull_face_off, s.hull_face_idx = np.zeros((0, 3)), np.zeros(1, np.int32), np.zeros(0, np.int32)
    mass = np.concatenate([[0.0], r.uniform(500.0, 1500.0, n)])
    v = np.concatenate([np.zeros((1, 3)), r.normal(0, 0.2, (n, 3)) + (0.0, -0.5, 0.0)])
    w = np.concatenate([np.zeros((1, 3)), r.normal(0, 0.3, (n, 3))])
    _bodies(s, np.arange(n + 1, dtype=np.int32), np.array([sc.KINEMATIC] + [0] * n, np.int32), mass,
            np.concatenate([[(0.0, -0.5, 0.0)], origin]), np.concatenate([np.eye(3)[None], basis]), v, w)
    s = s.rounded(c["bits"]) if c["bits"] == 32 else s
    # each body above its support: the floor, or the body one level down in its column
    up = np.arange(1, n + 1)
    low = np.where(level == 0, 0, up - cols)
    normal = np.array([0.0, 1.0, 0.0]) + r.normal(0, 0.01, (n, 3))
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    t0 = np.cross(normal, (1.0, 0.0, 0.0))
    t0 /= np.linalg.norm(t0, axis=1, keepdims=True)
    t1 = np.cross(normal, t0)
    slots = np.zeros((n, 8, 19))
    slots[:, 4:, 12] = 1e30 if c["bits"] == 32 else 1e100
    for k, (sx, sz) in enumerate(((-1, -1), (1, -1), (1, 1), (-1, 1))):
        corner = np.stack([sx * 0.4 * size[:, 0], np.full(n, -0.5), sz * 0.4 * size[:, 2]], axis=1)
        p = origin + np.einsum("nij,nj->ni", basis, corner)
        depth = -r.uniform(0.0, 0.01, n)
        la = corner
        lb = np.einsum("nji,nj->ni", s.basis[low], p - s.origin[low])
        for at, val in ((0, p), (3, normal), (6, la), (9, lb), (13, t0), (16, t1)):
            slots[:, k, at:at + 3] = val
        slots[:, k, 12] = depth
    slots = slots.astype(real).astype(np.float64)
    res = dict(res_a=up.astype(np.int32), res_b=low.astype(np.int32), point_size=np.full(n, 4, np.int32),
               friction=np.full(n, 0.5), restitution=np.zeros(n), slots=slots)
    return s, res


def _prepare_solve(c, seed):
    s, res = _contacts(c, seed)
    world = pg.GpuWorld(s, c["bits"], tuning="auto")
    world.set_results(res)
    dtype = np.float32 if c["bits"] == 32 else np.float64
    return dict(family="solve", world=world, mode=MODES[c["mode"]],
                inputs={"lin_vel": _pinned(s.lin_vel.astype(dtype)), "ang_vel": _pinned(s.ang_vel.astype(dtype))},
                out=_buffers(s.n_bodies, dtype, ("lin_vel", "ang_vel")))


def _exact_solve(c, seed):
    """Sequential impulses over the contacts in their order: a contact of level l shares no moving
    body with another of its level, and every contact below it in the column comes before it."""
    s, res = _contacts(c, seed)
    n, dt, iters = c["n"], s.dt, s.iterations
    a, b, slots = res["res_a"], res["res_b"], res["slots"]
    size, mass = s.shape_param, s.mass
    im = np.where(mass > 0, 1.0 / np.maximum(mass, 1e-30), 0.0)
    d = np.stack([size[:, 1] ** 2 + size[:, 2] ** 2, size[:, 0] ** 2 + size[:, 2] ** 2, size[:, 0] ** 2 + size[:, 1] ** 2], 1)
    inv = 12.0 * im[:, None] / d
    inv = np.einsum("nij,nj,nkj->nik", s.basis, inv, s.basis)
    pts = slots[:, :4]
    nrm, t0, t1, depth = pts[:, :, 3:6], pts[:, :, 13:16], pts[:, :, 16:19], pts[:, :, 12]
    ra = np.einsum("nij,nkj->nki", s.basis[a], pts[:, :, 6:9])
    rb = np.einsum("nij,nkj->nki", s.basis[b], pts[:, :, 9:12])
    ia, ib = inv[a], inv[b]

    def effective(u):
        xa, xb = np.cross(ra, u), np.cross(rb, u)
        return 1.0 / ((im[a] + im[b])[:, None] + np.einsum("nki,nij,nkj->nk", xa, ia, xa) + np.einsum("nki,nij,nkj->nk", xb, ib, xb))

    jn, j0, j1 = effective(nrm), effective(t0), effective(t1)
    rhs = -0.2 * np.maximum(depth, -0.3) / dt * jn
    v, w = s.lin_vel.copy(), s.ang_vel.copy()
    acc = np.zeros((3, n, 4))
    cols = int((b == 0).sum())
    levels = [np.arange(k, min(k + cols, n)) for k in range(0, n, cols)]
    for _ in range(iters):
        for i in levels:
            A, B = a[i], b[i]
            moves = (B > 0)[:, None]
            for k in range(4):
                vr = v[A] + np.cross(w[A], ra[i, k]) - v[B] - np.cross(w[B], rb[i, k])
                dn = rhs[i, k] - np.einsum("ni,ni->n", nrm[i, k], vr) * jn[i, k]
                dn = np.maximum(dn, -acc[0, i, k])
                acc[0, i, k] += dn
                u0 = acc[1, i, k] - np.einsum("ni,ni->n", t0[i, k], vr) * j0[i, k]
                u1 = acc[2, i, k] - np.einsum("ni,ni->n", t1[i, k], vr) * j1[i, k]
                with np.errstate(divide="ignore", invalid="ignore"):
                    f = 0.5 * acc[0, i, k] / np.sqrt(u0 * u0 + u1 * u1)
                f = np.where(f < 1, f, 1.0)
                u0, u1 = u0 * f, u1 * f
                imp = dn[:, None] * nrm[i, k] + (u0 - acc[1, i, k])[:, None] * t0[i, k] + (u1 - acc[2, i, k])[:, None] * t1[i, k]
                acc[1, i, k], acc[2, i, k] = u0, u1
                v[A] += imp * im[A][:, None]
                w[A] += np.einsum("nij,nj->ni", ia[i], np.cross(ra[i, k], imp))
                v[B] -= np.where(moves, imp * im[B][:, None], 0.0)
                w[B] -= np.where(moves, np.einsum("nij,nj->ni", ib[i], np.cross(rb[i, k], imp)), 0.0)
    return {"lin_vel": v, "ang_vel": w}
