"""The work that a user of this library has it do, as cases that can be timed.

Each case goes through the public Python objects over the C ABI
(diomedes_gb300.compute) and is one pass of what a host program does again
and again: a demo's frame through the reference-mirror calls, a detection
query, a solve of rows that the caller prepared, or a rollout of a
device-resident world -- poses and velocities set to a recorded frame (one
upload of motion records), a few steps, and the motion records read back, as
a planner or a learner does with a batch of scenes and as the demos' frame
loop does with one.  Sizes, options and distributions are those of
diomedes_gb300/scenes.py, the tests and bench.py.

The topology of a case (scene sizes, chain lengths, shape kinds) comes from
the case alone and the values (positions, orientations, velocities, sizes)
from the seed, so outputs of two seeds have the same shapes.
"""
import numpy as np
import torch

from diomedes_gb300 import abi, compute, scenes
from diomedes_gb300 import physics as ph

ICO = scenes.icosphere42()
TET = scenes.regular_tetrahedron(0.4)
NO_ROT = np.array([0.0, 0.0, 0.0, 1.0], np.float32)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference demos' frame (demos/avbd_box): a few dozen bodies in a
        # box through the mirror calls, host arrays in and out; all latency
        {"name": "demo_frame_47", "kind": "demo", "n": 47},
        # a collision query on a dense packing of cubes, spheres and hulls
        # through NarrowPhaseCompute: pairs and all contact slots read back
        {"name": "detect_1617", "kind": "detect", "nx": 11, "ny": 7, "nz": 21},
        # AvbdCompute.submit / read: rows prepared by the caller (stacks of
        # cubes, four rows a contact, ropes between the stacks)
        {"name": "solve_5005", "kind": "solve", "columns": 715, "height": 7},
        # the smallest resident world: the 10-level pyramid, 8-contact
        # manifold, one step a frame as an interactive program runs it
        {"name": "pyramid_55", "kind": "pyramid", "levels": 10, "per_pair": 8, "steps": 1},
        # a game-sized scene of mixed convex bodies, one step a frame
        {"name": "pile_901", "kind": "pile", "n": 901, "precision": "f32", "steps": 1},
        # one scene beyond a CTA's shared memory, contact-dense: 32 x 8 x 32 cubes
        {"name": "field_8192", "kind": "field", "nx": 32, "ny": 8, "nz": 32, "mode": "jacobi", "steps": 2},
        # the large mixed pile: GJK and EPA at scale
        {"name": "pile_50000", "kind": "pile", "n": 50000, "precision": "f32", "steps": 2},
        # the largest single scene, FP64 poses and FP32 rows
        {"name": "wall_400x500_split", "kind": "wall", "cols": 400, "rows": 500, "spheres": 1000, "steps": 1},
        # a small batch of jointed scenes (an evaluation run, a few seeds)
        {"name": "batch_33", "kind": "batch", "scenes": 33, "precision": "f32", "mode": "jacobi", "steps": 4},
        # the headline batch: 1024 scenes of 16 to 2048 bodies, a control
        # step of four physics steps
        {"name": "batch_1024", "kind": "batch", "scenes": 1024, "precision": "f32", "mode": "jacobi", "steps": 4},
        # the same work in split precision
        {"name": "batch_257_split", "kind": "batch", "scenes": 257, "precision": "split", "mode": "jacobi",
         "steps": 4},
        # the coloured Gauss-Seidel schedule on a batch
        {"name": "batch_150_colored", "kind": "batch", "scenes": 150, "precision": "f32", "mode": "colored",
         "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["demo", "detect", "solve", "pyramid", "pile", "pile", "field", "wall", "batch", "batch", "batch"])
    if kind == "demo":
        return {"kind": kind, "n": _log(rng, 8, 500)}
    if kind == "detect":
        return {"kind": kind, "nx": _log(rng, 2, 20), "ny": _log(rng, 2, 20), "nz": _log(rng, 2, 20)}
    if kind == "solve":
        return {"kind": kind, "columns": _log(rng, 4, 2000), "height": rng.randint(1, 9)}
    if kind == "pyramid":
        return {"kind": kind, "levels": rng.randint(2, 40), "per_pair": rng.choice([4, 8]), "steps": 1}
    if kind == "pile":
        n = _log(rng, 30, 50000)
        # the all-FP64 world is the reference run of error studies, at small sizes
        return {"kind": kind, "n": n, "precision": rng.choice(["f32", "f32", "split"] + ["f64"] * (n < 3000)),
                "steps": rng.choice([1, 2])}
    if kind == "field":
        return {"kind": kind, "nx": rng.randint(5, 32), "ny": rng.randint(2, 8), "nz": rng.randint(5, 32),
                "mode": rng.choice(["jacobi", "jacobi", "colored"]), "steps": rng.choice([1, 2])}
    if kind == "wall":
        cols, rows = _log(rng, 20, 400), _log(rng, 20, 400)
        return {"kind": kind, "cols": cols, "rows": rows, "spheres": _log(rng, 5, max(10, cols * rows // 160)),
                "steps": 1}
    return {"kind": kind, "scenes": _log(rng, 2, 1000), "precision": rng.choice(["f32", "f32", "split"]),
            "mode": rng.choice(["jacobi", "jacobi", "colored"]), "steps": rng.choice([1, 2, 4])}


def _topology(case):
    """Generator of what the case fixes and the seed does not vary."""
    text = "|".join(f"{k}={case[k]}" for k in sorted(case) if k != "name")
    return np.random.default_rng(list(text.encode()))


# -------------------------------------------------------------- body records
def _quats(rng, n):
    return scenes.random_quats(rng, n)


def _records(n):
    b, s = np.zeros(n, abi.BODY), np.zeros(n, abi.BODY_STATE)
    b["orientation"] = NO_ROT
    s["friction"] = 0.8
    return b, s


def _inverse(b, s, at, mass, moment):
    """Inverse mass and moment (k, 3) of bodies `at`; mass 0 is static."""
    mass = np.broadcast_to(np.asarray(mass, np.float64), (len(at),))
    live = mass > 0
    s["inv_mass"][at] = np.where(live, 1.0 / np.where(live, mass, 1.0), 0.0)
    m = np.broadcast_to(np.asarray(moment, np.float64).reshape(len(at), -1), (len(at), 3))
    s["inv_moment"][at, :3] = np.where(live[:, None], 1.0 / np.where(live[:, None], m, 1.0), 0.0)


def _spheres(b, s, at, radius, mass):
    b["shape"]["tag"][at] = abi.SPHERE
    b["shape"]["corners"][at, 0, 0] = radius
    mass = np.broadcast_to(np.asarray(mass, np.float64), (len(at),))
    _inverse(b, s, at, mass, 0.4 * mass * np.square(radius))


def _cubes(b, s, at, half, density=1000.0):
    half = np.broadcast_to(np.asarray(half, np.float64), (len(at),))
    b["shape"]["tag"][at] = abi.CUBE
    b["shape"]["corners"][at, 0, :3] = half[:, None]
    mass = density * 8 * half ** 3
    _inverse(b, s, at, mass, 2.0 / 3.0 * mass * half ** 2)


def _boxes(b, s, at, half, density):
    b["shape"]["tag"][at] = abi.BOX
    b["shape"]["corners"][at, 0, :3] = half
    mass = density * 8 * half.prod(1)
    q = half ** 2
    _inverse(b, s, at, mass, mass[:, None] / 3.0 * (q.sum(1, keepdims=True) - q))


def _hulls(b, s, at, radius, density):
    """42-vertex icosphere hulls; returns their vertices for the pool."""
    k = len(ICO)
    b["shape"]["tag"][at] = abi.HULL
    b["shape"]["pad"][at, 0] = np.arange(len(at)) * k
    b["shape"]["pad"][at, 1] = k
    mass = density * 4.0 / 3.0 * np.pi * radius ** 3
    _inverse(b, s, at, mass, 0.4 * mass * radius ** 2)
    v = np.zeros((len(at), k, 4), np.float32)
    v[:, :, :3] = ICO[None] * radius[:, None, None]
    return v.reshape(-1, 4)


def _tetrahedra(b, s, at, density):
    b["shape"]["tag"][at] = abi.TETRAHEDRON
    b["shape"]["corners"][at, :, :3] = TET
    mass = density * 0.4 ** 3 / (6 * 2 ** 0.5)
    _inverse(b, s, at, mass, 0.4 * mass * np.square(TET).sum(1).max())


# -------------------------------------------------------------------- scenes
class _Scene:
    def __init__(self, b, s, options, joints=None, offsets=None, containers=None, hull=None, per_body=(8, 16)):
        self.b, self.s, self.options, self.joints, self.offsets = b, s, options, joints, offsets
        self.containers, self.hull, self.per_body = containers or [scenes.ground()], hull, per_body


def _pyramid(case, rng):
    levels = case["levels"]
    k = np.repeat(np.arange(levels), levels - np.arange(levels))
    i = np.concatenate([np.arange(levels - v) for v in range(levels)])
    b, s = _records(len(k))
    b["position"][:, 0] = (i - (levels - k - 1) / 2.0) * 1.01 + rng.uniform(-2e-3, 2e-3, len(k))
    b["position"][:, 1] = 0.51 + k * 1.01
    _cubes(b, s, np.arange(len(k)), 0.5)
    o = ph.avbd_options(gravity=(0, -9.81, 0), alpha=0.95, beta_lin=1e5, penalty_min=1e4, friction=0.5)
    return _Scene(b, s, o, per_body=(64, 200))


def _field(case, rng):
    dims = (case["nx"], case["ny"], case["nz"])
    g = np.stack(np.meshgrid(*map(np.arange, dims), indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    b, s = _records(len(g))
    g[:, [0, 2]] -= (np.array(dims)[[0, 2]] - 1) / 2
    b["position"][:, :3] = g * 0.6 + [0, 2.0, 0] + rng.uniform(-0.05, 0.05, g.shape)
    b["orientation"] = _quats(rng, len(g))
    _cubes(b, s, np.arange(len(g)), 0.25)
    return _Scene(b, s, ph.avbd_options(gravity=(0, -9.81, 0), friction=0.6), per_body=(24, 32))


def _pile(case, rng):
    """40% boxes, 40% hulls, 20% tetrahedra at the 50,000-body pile's density."""
    n = case["n"]
    extent = 40.0 * (n / 50000.0) ** (1.0 / 3.0)
    kinds = _topology(case).permutation(np.repeat([0, 1, 2], [int(0.4 * n), int(0.4 * n), n - 2 * int(0.4 * n)]))
    b, s = _records(n)
    b["position"][:, :3] = rng.uniform(0, extent, (n, 3)) + [-extent / 2, 1.0, -extent / 2]
    b["orientation"] = _quats(rng, n)
    rho = rng.uniform(500.0, 2000.0, n)
    box, ico, tet = (np.flatnonzero(kinds == k) for k in range(3))
    _boxes(b, s, box, np.exp(rng.normal(np.log(0.25), 0.3, (len(box), 3))), rho[box])
    hull = _hulls(b, s, ico, np.exp(rng.normal(np.log(0.25), 0.3, len(ico))), rho[ico])
    _tetrahedra(b, s, tet, rho[tet])
    return _Scene(b, s, ph.avbd_options(gravity=(0, -9.81, 0), dt=1.0 / 120.0, iterations=12), hull=hull,
                  per_body=(8, 16))


def _wall(case, rng):
    """Bricks 0.4 x 0.2 x 0.2 m in running bond and spheres thrown at them.
    The wall stands at the origin: motion records are FP32, and the rollout
    restarts from them."""
    cols, rows, k = case["cols"], case["rows"], case["spheres"]
    r, c = (v.ravel().astype(np.float64) for v in np.meshgrid(np.arange(rows), np.arange(cols), indexing="ij"))
    n = len(r)
    b, s = _records(n + k)
    b["position"][:n, 1] = 0.1 + 0.2 * r
    b["position"][:n, 2] = (c - (cols - 1) / 2.0) * 0.4 + 0.2 * (r % 2)
    _boxes(b, s, np.arange(n), np.tile([0.1, 0.1, 0.2], (n, 1)), np.full(n, 2000.0))
    ball = np.arange(n, n + k)
    yaw, pitch = np.radians(rng.uniform(-5, 5, (2, k)))
    # the front of the throw has just reached the wall
    b["position"][ball, 0] = -0.42 - rng.uniform(0, 10, k)
    b["position"][ball, 1] = rng.uniform(1.0, max(1.5, rows * 0.16), k)
    b["position"][ball, 2] = rng.uniform(-cols * 0.15, cols * 0.15, k)
    s["vel"][ball, :3] = 30.0 * np.stack([np.cos(pitch) * np.cos(yaw), np.sin(pitch), np.cos(pitch) * np.sin(yaw)], 1)
    _spheres(b, s, ball, 0.3, 2000.0 * 4.0 / 3.0 * np.pi * 0.027)
    return _Scene(b, s, ph.avbd_options(gravity=(0, -9.81, 0), dt=1.0 / 120.0, iterations=15), per_body=(6, 12))


def _batch(case, rng):
    """Independent scenes of log-uniform sizes in [16, 2048]: rope, ball-socket
    and spring chains of 2 to 20 bodies hung from static anchors, and up to
    200 loose boxes (scenes.joint_scene, built for all scenes at once)."""
    top, count = _topology(case), case["scenes"]
    sizes = np.floor(np.exp(top.uniform(np.log(16), np.log(2048), count))).astype(int)
    loose = top.integers(0, np.minimum(200, sizes // 2) + 1)
    lengths, owner = [], []
    for k in range(count):
        budget = int(sizes[k] - loose[k])
        ends = np.cumsum(top.integers(2, 21, budget // 2 + 1))
        m = int(np.searchsorted(ends, budget)) + 1
        one = np.diff(np.minimum(ends[:m], budget), prepend=0)
        lengths.append(one)
        owner.append(np.full(m, k))
    slot = np.concatenate([np.arange(len(v)) for v in lengths])
    length, owner = np.concatenate(lengths), np.concatenate(owner)
    offsets = np.concatenate([[0], np.cumsum(sizes)])
    before = np.cumsum(length) - length  # chain bodies of all earlier chains
    loose_before = np.cumsum(loose) - loose
    base = before + loose_before[owner]  # loose boxes of earlier scenes lie between
    grid = np.ceil(np.sqrt(np.maximum(1.0, (sizes - loose) / 8.0)))
    g = grid[owner]
    cx, cz = (slot % g - g / 2.0) * 2.0, (slot // g - g / 2.0) * 2.0
    cy = 12.0 + rng.uniform(0.0, 2.0, len(length))
    n = int(offsets[-1])
    b, s = _records(n)
    chain = np.repeat(np.arange(len(length)), length)
    k = (np.arange(len(chain)) - before[chain]).astype(np.float64)
    at = base[chain] + k.astype(int)
    kind = slot[chain] % 3
    p = np.stack([cx[chain], cy[chain], cz[chain]], 1)
    p[:, 0] += np.select([kind == 0, kind == 1], [0.14 * k, 0.2 * k], 0.0)
    p[:, 1] -= np.select([kind == 0, kind == 2], [0.14 * k, 0.5 * k], 0.0)
    p[:, 2] += np.where(kind == 2, 0.05 * k, 0.0)
    b["position"][at, :3] = p
    _spheres(b, s, at, 0.05, np.where(k > 0, 1.0, 0.0))
    link = k > 0
    j = np.zeros(int(link.sum()), abi.CONSTRAINT)
    j["a"], j["b"] = at[link] - 1, at[link]
    kj = kind[link]
    j["kind"] = np.choose(kj, [abi.ROPE, abi.BALL_SOCKET, abi.SPRING])
    j["anchor_a"][:, 0] = np.where(kj == 1, 0.1, 0.0)
    j["anchor_b"][:, 0] = np.where(kj == 1, -0.1, 0.0)
    j["anchor_a"][:, 3] = np.choose(kj, [0.2, 0.0, 0.5])
    j["anchor_b"][:, 3] = 1000.0
    scene = np.repeat(np.arange(count), loose)
    i = np.arange(len(scene)) - loose_before[scene]
    side = np.maximum(1, np.ceil(np.sqrt(loose))).astype(int)[scene]
    at = offsets[scene] + (sizes - loose)[scene] + i
    half = rng.uniform(0.1, 0.2, len(i))
    b["position"][at, 0] = grid[scene] + 4.0 + (i % side) * 0.5 + rng.uniform(-0.02, 0.02, len(i))
    b["position"][at, 1] = half + 0.02 + rng.uniform(0, 0.5, len(i))
    b["position"][at, 2] = -4.0 + (i // side) * 0.5
    _cubes(b, s, at, half)
    return _Scene(b, s, ph.avbd_options(gravity=(0, -9.81, 0)), joints=j, offsets=offsets.astype(np.uint32),
                  containers=[scenes.ground(1000.0)] * count, per_body=(2, 4))


BUILD = {"pyramid": _pyramid, "field": _field, "pile": _pile, "wall": _wall, "batch": _batch}
PRECISION = {"f32": abi.PREC_F32, "split": abi.PREC_SPLIT, "f64": abi.PREC_F64}
WARM_STEPS = 24  # into the run: contacts formed, rows warm-started


def _pinned_motion(n):
    return torch.empty((n, 16), dtype=torch.float32, pin_memory=True).numpy()


def _prepare_world(case, rng):
    sc = BUILD[case["kind"]](case, rng)
    n, o = len(sc.b), sc.options
    cap = compute.capacity(n, max_pairs=max(1024, sc.per_body[0] * n), max_contacts=max(4096, sc.per_body[1] * n),
                           max_joints=max(1, 0 if sc.joints is None else len(sc.joints)),
                           max_scenes=len(sc.containers),
                           max_hull_vertices=max(1, 0 if sc.hull is None else len(sc.hull)))
    per_pair = case.get("per_pair", 4)
    w = compute.World(cap, contacts_per_pair=per_pair,
                      precision=PRECISION["split" if case["kind"] == "wall" else case.get("precision", "f32")],
                      solver_mode=abi.SOLVER_COLORED if case.get("mode") == "colored" else abi.SOLVER_JACOBI)
    w.upload(sc.b, sc.s, constraints=sc.joints, scene_offsets=sc.offsets, containers=sc.containers,
             hull_vertices=sc.hull)
    w.step(o, 4 if case["kind"] == "wall" else WARM_STEPS)
    start, out = _pinned_motion(n), _pinned_motion(n)
    w.download_motion_into(start.view(abi.MOTION).reshape(n))
    return {"world": w, "options": o, "steps": case["steps"], "start": start.view(abi.MOTION).reshape(n),
            "motion": out.view(abi.MOTION).reshape(n), "out": out}


def _run_world(st):
    w = st["world"]
    w.set_motion(st["start"])
    w.step_async(st["options"], st["steps"])
    w.download_motion_into(st["motion"])
    return st["out"]


# ------------------------------------------------- the reference-mirror calls
def _prepare_demo(case, rng):
    """Cubes, tetrahedra and spheres with random velocities in a 2 m box (its
    size grows with the bodies), as demos/avbd_box sets them up."""
    n = case["n"]
    half = 2.0 * max(1.0, (n / 48.0) ** (1.0 / 3.0))
    side = int(np.ceil(n ** (1.0 / 3.0)))
    cell = _topology(case).permutation(side ** 3)[:n]
    p = np.stack([cell % side, cell // side % side, cell // side ** 2], 1) + 0.5
    b, s = _records(n)
    b["position"][:, :3] = (p / side * 2.0 - 1.0) * (half - 0.25) + rng.uniform(-0.05, 0.05, (n, 3))
    s["vel"][:, :3] = rng.uniform(-0.9, 0.9, (n, 3))
    s["ang"][:, :3] = rng.uniform(-1.2, 1.2, (n, 3))
    corners = np.array([(0.0, -0.707, -1.0), (0.866025, -0.707, 0.5), (-0.866025, -0.707, 0.5), (0.0, 0.707, 0.0)])
    i = np.arange(n)
    cube, tet, ball = i[: n // 8], i[n // 8: n // 4], i[n // 4:]
    b["shape"]["tag"][cube], b["shape"]["corners"][cube, 0, :3] = abi.CUBE, 0.4
    _inverse(b, s, cube, 1.0, np.full(len(cube), 2.0 / 3.0 * 0.16))
    b["shape"]["tag"][tet], b["shape"]["corners"][tet, :, :3] = abi.TETRAHEDRON, corners * 0.55
    _inverse(b, s, tet, 1.0, np.full(len(tet), 0.4 * (0.55 ** 2) * 1.5))
    _spheres(b, s, ball, 0.3, 1.0)
    pairs, rows = 64 * n + 64, 64 * n + 256
    st = {"kind": "demo", "n": n, "b": b, "s": s, "options": ph.avbd_options(alpha=0.8),
          "container": ph.container((0, 0, 0), half), "prev": None, "narrow": compute.NarrowPhaseCompute(n, pairs),
          "avbd": compute.AvbdCompute(n, rows, max_pairs=pairs), "joints": np.zeros(0, abi.CONSTRAINT),
          "lambda": np.zeros((rows, 3), np.float32), "rows": np.zeros(rows, abi.CONTACT)}
    st["run_options"] = ph.run_options(st["options"])
    # the previous frame's rows, which a running demo has in hand
    r, rows = _demo_frame(st)
    rows = rows.copy()
    rows["lambda"][:, :3], rows["penalty"][:, :3] = r["lambda"], r["penalty"]
    st["prev"] = rows
    return st


def _demo_frame(st):
    """One frame of the demos: detect, prepare the rows, solve, read back."""
    narrow, avbd, b = st["narrow"], st["avbd"], st["b"]
    narrow.submit_broad(b)
    count = narrow.read_pair_count()
    narrow.submit_narrow(count)
    slots = compute.decode_contacts(narrow.read())
    rows, offsets, indices = avbd.prepare_contacts(b, st["s"], slots, st["prev"], st["container"], st["options"])
    return avbd.run(st["s"], b["position"][:, :3], b["orientation"], rows, st["joints"], offsets, indices,
                    st["run_options"]), rows


def _run_demo(st):
    r, rows = _demo_frame(st)
    # the rows' number depends on the values: they come back in buffers of a fixed size
    m = len(rows)
    st["lambda"][:m], st["lambda"][m:] = r["lambda"], 0.0
    return {"positions": r["positions"], "orientations": r["orientations"], "velocities": r["velocities"],
            "angular_velocities": r["angular_velocities"], "rows": m, "lambda": st["lambda"]}


def _prepare_detect(case, rng):
    """A dense packing on a 0.48 m grid: every neighbour's box overlaps at
    every orientation and nothing further does, so the number of pairs is
    the case's; whether and where a pair touches is the values'."""
    dims = (case["nx"], case["ny"], case["nz"])
    g = np.stack(np.meshgrid(*map(np.arange, dims), indexing="ij"), -1).reshape(-1, 3)
    n = len(g)
    kinds = _topology(case).integers(0, 3, n)
    b, s = _records(n)
    b["position"][:, :3] = g * 0.48 + rng.uniform(-0.008, 0.008, (n, 3))
    b["orientation"] = _quats(rng, n)
    cube, ball, ico = (np.flatnonzero(kinds == k) for k in range(3))
    _cubes(b, s, cube, 0.25)
    _spheres(b, s, ball, rng.uniform(0.25, 0.3, len(ball)), 100.0)
    hull = _hulls(b, s, ico, rng.uniform(0.29, 0.33, len(ico)), np.full(len(ico), 1000.0))
    nc = compute.NarrowPhaseCompute(n, 13 * n, max_hull_vertices=max(1, len(hull)))
    if len(hull):
        nc.set_hull_vertices(hull)
    return {"kind": "detect", "narrow": nc, "b": b}


def _run_detect(st):
    nc = st["narrow"]
    nc.submit_broad(st["b"])
    count = nc.read_pair_count()
    pairs = nc.read_pairs(count)
    nc.submit_narrow(count)
    slots = nc.read()
    return {"pairs": pairs.view(np.uint32), "valid": slots["valid"], "normal": slots["normal"],
            "depth": slots["depth"], "point_a": slots["point_a"], "point_b": slots["point_b"]}


def _stack_rows(case, rng):
    """Columns of unit cubes, four rows a contact, and ropes between the tops
    of neighbouring columns, in the arrays that AvbdCompute.submit takes."""
    cols, h = case["columns"], case["height"]
    n = cols * h
    col, lev = np.arange(n) // h, np.arange(n) % h
    side = int(np.ceil(np.sqrt(cols)))
    b, s = _records(n)
    pos = np.stack([(col % side) * 2.0, 0.5 + lev, (col // side) * 2.0], 1) + rng.uniform(-0.01, 0.01, (n, 3))
    rot = NO_ROT + np.concatenate([rng.uniform(-0.01, 0.01, (n, 3)), np.zeros((n, 1))], 1)
    rot /= np.linalg.norm(rot, axis=1, keepdims=True)
    _cubes(b, s, np.arange(n), 0.5)
    for f, v in (("vel", 0.1), ("ang", 0.1), ("prev_vel", 0.1)):
        s[f][:, :3] = rng.uniform(-v, v, (n, 3))
    # pair rows (lower cube, upper cube) in order, then the floor rows
    low = np.flatnonzero(lev < h - 1)
    floor = np.flatnonzero(lev == 0)
    a = np.repeat(np.concatenate([low, floor]), 4)
    pair = np.arange(len(a)) < 4 * len(low)
    m = len(a)
    c = np.zeros(m, abi.CONTACT)
    c["a"], c["b"], c["friction"] = a, np.where(pair, a + 1, abi.CONTAINER), 0.8
    corner = np.tile([(0.5, 0.5), (-0.5, 0.5), (-0.5, -0.5), (0.5, -0.5)], (m // 4, 1))
    c["normal"][:, 1] = np.where(pair, -1.0, 1.0)
    c["tangent1"][:, 2], c["tangent2"][:, 0] = np.where(pair, -1.0, 1.0), np.where(pair, -1.0, 1.0)
    c["r_a"][:, [0, 2]], c["r_a"][:, 1] = corner + rng.uniform(-0.02, 0.02, (m, 2)), np.where(pair, 0.5, -0.5)
    c["r_b"][:, [0, 2]] = np.where(pair[:, None], corner + rng.uniform(-0.02, 0.02, (m, 2)), 0.0)
    c["r_b"][:, 1] = np.where(pair, -0.5, 0.0)
    c["c0"][:, 0] = 0.01 - rng.uniform(0.0, 0.02, m)
    c["penalty"][:, :3] = 10.0 ** rng.uniform(3, 5, (m, 3))
    c["lambda"][:, 0] = -rng.uniform(0, 3000, m)
    c["lambda"][:, 1:3] = rng.uniform(-300, 300, (m, 2))
    body = np.stack([c["a"], c["b"]], 1).astype(np.int64).ravel()
    row = np.repeat(np.arange(m), 2)
    keep = body < n
    order = np.argsort(body[keep], kind="stable")
    offsets = np.concatenate([[0], np.cumsum(np.bincount(body[keep], minlength=n))]).astype(np.uint32)
    j = np.zeros(cols - 1, abi.CONSTRAINT)
    j["a"] = np.arange(cols - 1) * h + h - 1
    j["b"] = j["a"] + h
    j["kind"] = abi.ROPE
    j["anchor_a"][:, 3], j["anchor_b"][:, 3] = 1.9, 1000.0
    return {"state": s, "positions": pos.astype(np.float32), "orientations": rot.astype(np.float32), "contacts": c,
            "constraints": j, "offsets": offsets, "indices": row[keep][order].astype(np.uint32)}


def _solve_options():
    return ph.run_options(ph.avbd_options(gravity=(0, -9.81, 0)))


def _prepare_solve(case, rng):
    x = _stack_rows(case, rng)
    n, m = len(x["state"]), len(x["contacts"])
    args = [x[k] for k in ("state", "positions", "orientations", "contacts", "constraints", "offsets", "indices")]
    return {"kind": "solve", "avbd": compute.AvbdCompute(n, m, max_joints=max(1, len(x["constraints"]))),
            "args": args + [_solve_options()]}


def _run_solve(st):
    st["avbd"].submit(*st["args"])
    return st["avbd"].read()


# ------------------------------------------------------------------ interface
def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    made = {"demo": _prepare_demo, "detect": _prepare_detect, "solve": _prepare_solve}.get(case["kind"], _prepare_world)
    return made(case, rng)


def run(state):
    return {"demo": _run_demo, "detect": _run_detect, "solve": _run_solve}.get(state.get("kind"), _run_world)(state)


def _bodies(case):
    k = case["kind"]
    if k == "pyramid":
        return case["levels"] * (case["levels"] + 1) // 2
    if k in ("field", "detect"):
        return case["nx"] * case["ny"] * case["nz"]
    if k == "solve":
        return case["columns"] * case["height"]
    if k == "wall":
        return case["cols"] * case["rows"] + case["spheres"]
    if k == "batch":
        top = _topology(case)
        return int(np.floor(np.exp(top.uniform(np.log(16), np.log(2048), case["scenes"]))).sum())
    return case["n"]


# contact rows a body carries in a step, about, and the solver's iterations
ROWS = {"pyramid": 7.0, "field": 6.0, "pile": 1.0, "wall": 8.0, "batch": 0.5, "demo": 1.5, "solve": 4.0}
ITERATIONS = {"pile": 12, "wall": 15}


def work(case):
    """Bytes: per pass every body's motion record in and out, and per step its
    shape, mass, pose and velocities read once and pose and velocities
    written once, each contact row's payload and duals written and read once
    (the next step's warm start), each joint's record read once.  Operations:
    per step and iteration a 6 x 6 solve a body (~350), three stamps of 27
    entries a row and body (~700 both sides), a dual update a row (~200), and
    one to three stamps a joint and body."""
    n, k = _bodies(case), case["kind"]
    if k == "detect":
        x, y, z = case["nx"], case["ny"], case["nz"]
        pairs = ((3 * x - 2) * (3 * y - 2) * (3 * z - 2) - n) // 2
        return {"bytes": 112 * n + 8 * pairs + 320 * pairs, "flops": 300 * n + 1500 * pairs}
    rows = ROWS[k] * n
    joints = 0.8 * n if k == "batch" else (case["columns"] - 1 if k == "solve" else 0)
    flops = ITERATIONS.get(k, 10) * (350 * n + 900 * rows + 400 * joints) + 300 * n + 500 * rows
    if k == "solve":
        return {"bytes": (80 + 28 + 64) * n + (144 + 24 + 12) * rows + 48 * joints, "flops": flops}
    if k == "demo":
        return {"bytes": (112 + 80 + 64) * n + (80 + 144 * 2 + 24) * rows, "flops": flops}
    wide = 2 if k == "wall" or case.get("precision") in ("split", "f64") else 1
    step = n * (80 + 20 + wide * (80 + 80)) + rows * (88 + 32 * wide + 24) + 48 * joints
    return {"bytes": 128 * n + case["steps"] * step, "flops": case["steps"] * flops}


# ------------------------------------------------------------- 64-bit results
def _cross(a, b):
    return torch.linalg.cross(a, b)


def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def _conj(q):
    return q * torch.tensor([-1.0, -1.0, -1.0, 1.0], dtype=q.dtype)


def _turn(q, v):
    u, w = q[..., :3], q[..., 3:]
    return v * (w * w - (u * u).sum(-1, keepdim=True)) + 2 * u * (u * v).sum(-1, keepdim=True) + 2 * w * _cross(u, v)


def _advance(q, d):
    p = q + 0.5 * _qmul(torch.cat([d, torch.zeros_like(d[..., :1])], -1), q)
    return p / p.norm(dim=-1, keepdim=True)


def _angle(to, frm):
    return 2 * _qmul(to, _conj(frm))[..., :3]


def exact(case, seed):
    """The solve of caller-prepared rows in 64 bits: inertial target and warm
    start, `iterations` Jacobi sweeps of the 6 x 6 body systems with the row
    forces' cone clamp and the dual and penalty update, velocities.  The
    other cases decide by branches (which pairs touch, which face is
    nearest) before anything is computed, so they have no such value."""
    if case["kind"] != "solve":
        return None
    x = _stack_rows(case, np.random.default_rng([seed, 77]))
    o = _solve_options()
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64))  # noqa: E731
    f = lambda v: float(np.float32(v))  # noqa: E731
    dt, alpha, beta, kmax, g = f(o.dt), f(o.alpha), f(o.beta_lin), f(o.penalty_max), t(list(o.gravity))
    s, c, j = x["state"], x["contacts"], x["constraints"]
    p0, q0 = t(x["positions"]), t(x["orientations"])
    vel, ang, prev = (t(s[k][:, :3]) for k in ("vel", "ang", "prev_vel"))
    mass, moment = 1.0 / t(s["inv_mass"])[:, None], 1.0 / t(s["inv_moment"][:, :3])
    n, m = len(p0), len(c)
    # inertial target, and a start moved by the part of gravity that acted last step
    target, target_q = p0 + vel * dt + g * dt * dt, _advance(q0, ang * dt)
    gm = g.norm()
    weight = (((vel - prev) / dt) @ (g / gm) / gm).clamp(0, 1)[:, None]
    p, q = p0 + vel * dt + g * weight * dt * dt, target_q.clone()
    a = torch.from_numpy(c["a"].astype(np.int64))
    paired = torch.from_numpy(c["b"] != abi.CONTAINER)
    b = torch.where(paired, torch.from_numpy(c["b"].astype(np.int64)), a)
    dirs = torch.stack([t(c[k][:, :3]) for k in ("normal", "tangent1", "tangent2")], 1)  # (m, 3, 3)
    ra, rb, c0 = t(c["r_a"][:, :3]), t(c["r_b"][:, :3]), t(c["c0"][:, :3]) * (1 - alpha)
    mu, lam, pen = t(c["friction"]), t(c["lambda"][:, :3]), t(c["penalty"][:, :3])
    has = paired[:, None].to(torch.float64)

    def spans():
        """World lever arms, Jacobians' angular parts and constraint values."""
        wa, wb = _turn(q[a], ra), _turn(q[b], rb)
        ja, jb = (_cross(w[:, None].expand_as(dirs), dirs) for w in (wa, wb))
        da, db = (p - p0), _angle(q, q0)
        value = c0 + (dirs * da[a][:, None]).sum(-1) + (ja * db[a][:, None]).sum(-1)
        value = value - has * ((dirs * da[b][:, None]).sum(-1) + (jb * db[b][:, None]).sum(-1))
        return ja, jb, value

    def forces(value):
        f0 = (pen[:, 0] * value[:, 0] + lam[:, 0]).clamp(max=0)
        ft = pen[:, 1:] * value[:, 1:] + lam[:, 1:]
        size, most = ft.norm(dim=1), f0.abs() * mu
        k = torch.where(size > most, most / size.clamp(min=1e-300), torch.ones_like(size))
        return torch.cat([f0[:, None], ft * k[:, None]], 1), size <= most

    ja_, jb_ = torch.from_numpy(j["a"].astype(np.int64)), torch.from_numpy(j["b"].astype(np.int64))
    anc_a, anc_b = t(j["anchor_a"][:, :3]), t(j["anchor_b"][:, :3])
    rest, stiff = t(j["anchor_a"][:, 3]), t(j["anchor_b"][:, 3])
    eye = torch.eye(3, dtype=torch.float64)
    for _ in range(o.iterations):
        H = torch.zeros(n, 6, 6, dtype=torch.float64)
        H[:, :3, :3] = eye * (mass / (dt * dt))[:, :, None]
        H[:, 3:, 3:] = eye * (moment / (dt * dt))[:, :, None]
        G = torch.cat([mass / (dt * dt) * (p - target), moment / (dt * dt) * _angle(q, target_q)], 1)
        ja, jb, value = spans()
        fr, _ = forces(value)
        for body, J, on in ((a, torch.cat([dirs, ja], 2), torch.ones_like(has)),
                            (b, -torch.cat([dirs, jb], 2), has)):
            J = J * on[:, :, None]
            H.index_add_(0, body, torch.einsum("mrx,mry,mr->mxy", J, J, pen))
            G.index_add_(0, body, torch.einsum("mrx,mr->mx", J, fr))
        if len(j):
            wa, wb = _turn(q[ja_], anc_a), _turn(q[jb_], anc_b)
            d = p[ja_] + wa - p[jb_] - wb
            ln = d.norm(dim=1)
            on = ((ln > 1e-6) & (ln > rest)).to(torch.float64)
            u = d / ln.clamp(min=1e-300)[:, None]
            for body, arm, sign in ((ja_, wa, 1.0), (jb_, wb, -1.0)):
                J = torch.cat([sign * u, _cross(arm, sign * u)], 1)
                H.index_add_(0, body, torch.einsum("mx,my,m->mxy", J, J, stiff * on))
                G.index_add_(0, body, J * (stiff * (ln - rest) * on)[:, None])
        dx = torch.linalg.solve(H, -G)
        p, q = p + dx[:, :3], _advance(q, dx[:, 3:])
        _, _, value = spans()
        lam, slip_free = forces(value)
        grown = (pen + beta * value.abs()).clamp(max=kmax)
        grow = torch.stack([lam[:, 0] < 0, slip_free, slip_free], 1)
        pen = torch.where(grow, grown, pen)
    return {"positions": p, "orientations": q, "velocities": (p - p0) / dt, "angular_velocities": _angle(q, q0) / dt,
            "prev_velocities": vel, "lambda": lam, "penalty": pen}
