"""The workloads this repository's step is timed on.

Each case is one pass as a program using the framework makes it: hand the world the state of this frame
(`World.set_state`), step it, read the new state back (`World.get_state`), or one gradient or query call.
Scenes are seeded and synthetic. Contacts exist from the first frame on: heaps are built in columns of
bodies that rest on one another with millimetre overlaps, as a settled pile does.

Kinds and what they stand for:
  stack     one small interactive scene: the reference's stack example (cubes on a floor)
  towers    many towers of cubes with mass ratio 1:100 at 50 substeps, the precision-stress workload
  heap      one scene of mixed hulls in a walled box (cube, icosahedron, 32-segment cylinder, 42-vertex
            icosphere), the plain form, from small scenes to thousands of bodies, in both precisions
  batch     many independent heaps of uneven size, a quarter of them with a hinge or spherical chain: the
            batched form, as a learning or sampling program steps it
  chains    joints only, collisions off: hinge, spherical and positional (spring) chains
  spheres   analytic spheres and compound bodies: the general narrowphase path
  dominoes  gradients of a loss on the last domino of a row (contacts on the tape)
  swing     gradients of a loss on the last link of a hinge or spherical chain (joints on the tape)
  queries   the broad-phase pair query and the transformed hulls of a large scene
"""
import math

import numpy as np

import sys
import os

sys.path.insert(0, os.path.join(os.getcwd(), "raw-physics_gb300"))

import rawphys  # noqa: E402
from rawphys import meshes as M  # noqa: E402
from rawphys import scenes as S  # noqa: E402

GRAVITY = 10.0
DT = 1.0 / 60.0
CELL = 1.75           # column spacing of a heap (metres): hulls of neighbouring columns are near but apart
LINK = (0.1, 0.3, 0.1)  # half extents of a chain link
JOINTS = ("hinge", "spherical", "positional")


def listed():
    return [
        # the smallest calls: the interactive ten-cube stack, once in each precision
        {"name": "stack10", "kind": "stack", "bodies": 10, "precision": "fp32", "substeps": 20},
        {"name": "stack10_fp64", "kind": "stack", "bodies": 10, "precision": "fp64", "substeps": 20},
        # the precision-stress towers: deep serial contact chains
        {"name": "towers96", "kind": "towers", "scenes": 96, "bodies": 64, "precision": "fp32", "substeps": 50},
        # one scene: a small heap, the plain form's 4096 bodies, and the exact build on an odd size
        {"name": "heap150", "kind": "heap", "bodies": 150, "precision": "fp32", "substeps": 20},
        {"name": "heap4096", "kind": "heap", "bodies": 4096, "precision": "fp32", "substeps": 20},
        {"name": "heap701_fp64", "kind": "heap", "bodies": 701, "precision": "fp64", "substeps": 20},
        # the batched form: a small batch and a large one
        {"name": "batch96", "kind": "batch", "scenes": 96, "most": 512, "precision": "fp32", "substeps": 20},
        {"name": "batch4096", "kind": "batch", "scenes": 4096, "most": 512, "precision": "fp32", "substeps": 20},
        # articulated bodies without collisions
        {"name": "chains768", "kind": "chains", "scenes": 768, "links": 33, "precision": "fp32", "substeps": 20},
        # spheres and compound bodies
        {"name": "spheres64", "kind": "spheres", "scenes": 64, "bodies": 11, "precision": "fp32", "substeps": 20},
        # gradients through contacts
        {"name": "dominoes24", "kind": "dominoes", "scenes": 24, "bodies": 12, "frames": 1, "substeps": 20},
        # queries between steps
        {"name": "queries20011", "kind": "queries", "bodies": 20011, "precision": "fp32"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["stack", "towers", "heap", "heap", "batch", "batch", "chains", "spheres", "dominoes", "swing", "queries"])
    precision = "fp64" if rng.random() < 0.25 else "fp32"
    substeps = rng.choice([10, 20, 20, 20, 25])
    if kind == "stack":
        return {"kind": kind, "bodies": _log(rng, 2, 40), "precision": precision, "substeps": substeps}
    if kind == "towers":
        return {"kind": kind, "scenes": _log(rng, 2, 96), "bodies": _log(rng, 8, 64), "precision": "fp32",
                "substeps": rng.choice([20, 50])}
    if kind == "heap":
        return {"kind": kind, "bodies": _log(rng, 20, 700 if precision == "fp64" else 4096), "precision": precision,
                "substeps": substeps}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 8, 64 if precision == "fp64" else 3000), "most": rng.choice([64, 200, 512]),
                "precision": precision, "substeps": min(substeps, 20)}
    if kind == "chains":
        return {"kind": kind, "scenes": _log(rng, 1, 768), "links": _log(rng, 4, 64), "precision": precision,
                "substeps": substeps}
    if kind == "spheres":
        return {"kind": kind, "scenes": _log(rng, 1, 64), "bodies": _log(rng, 3, 16), "precision": "fp32",
                "substeps": substeps}
    if kind == "dominoes":
        return {"kind": kind, "scenes": _log(rng, 1, 64), "bodies": rng.randint(4, 12), "frames": 1, "substeps": rng.choice([10, 20])}
    if kind == "swing":
        return {"kind": kind, "scenes": _log(rng, 1, 64), "links": rng.randint(3, 12), "frames": rng.randint(1, 2),
                "substeps": rng.choice([10, 20])}
    return {"kind": kind, "bodies": _log(rng, 300, 30000), "precision": "fp32"}


# -- scenes ---------------------------------------------------------------------------------------
def _qmul(a, b):
    ax, ay, az, aw = np.moveaxis(a, -1, 0)
    bx, by, bz, bw = np.moveaxis(b, -1, 0)
    return np.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by + ay * bw + az * bx - ax * bz,
                     aw * bz + az * bw + ax * by - ay * bx, aw * bw - ax * bx - ay * by - az * bz], -1)


def _matrix(q):
    x, y, z, w = np.moveaxis(q, -1, 0)
    return np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)], -1),
                     np.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)], -1),
                     np.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1)], -2)


def _arc(u, v):
    """Shortest-arc unit quaternion taking unit vector u to unit vector v."""
    q = np.concatenate([np.cross(u, v), [1.0 + float(np.dot(u, v))]])
    return q / np.linalg.norm(q) if np.linalg.norm(q) > 1e-6 else np.array([1.0, 0.0, 0.0, 0.0])


class _Shapes:
    """The four meshes: unique vertices, volume, and the rotation that puts a face down."""
    cached = None

    @classmethod
    def get(cls):
        if cls.cached is None:
            mesh = [M.MESHES[n]() for n in S.SHAPES]
            verts = [np.unique(m.positions.astype(np.float64), axis=0) for m in mesh]
            volume = np.array([M.hull_volume(m) for m in mesh])
            down = []
            for name, m in zip(S.SHAPES, mesh):
                a, b, c = m.positions[:3].astype(np.float64)
                n = np.cross(b - a, c - a)
                down.append(_arc(n / np.linalg.norm(n), np.array([0.0, -1.0, 0.0])) if name.startswith("ico")
                            else np.array([0.0, 0.0, 0.0, 1.0]))
            cls.cached = mesh, verts, volume, np.array(down)
        return cls.cached


def _heaps(sizes, links, seed, substeps):
    """Scenes of sizes[s] hulls each, in columns about four high on a floor inside four walls; links[s] > 0
    hangs a chain of that many links from an anchor above the heap."""
    rng = np.random.default_rng(seed)
    mesh, verts, volume, down = _Shapes.get()
    sizes, links = np.asarray(sizes), np.asarray(links)
    count = 5 + sizes + np.where(links > 0, links + 1, 0)
    start = np.concatenate([[0], np.cumsum(count)])
    N, K = int(start[-1]), len(sizes)
    f = {"scene": np.repeat(np.arange(K, dtype=np.int32), count), "mesh": np.zeros(N, np.int32), "scale": np.zeros((N, 3)),
         "pos": np.zeros((N, 3)), "rot": np.tile([0.0, 0.0, 0.0, 1.0], (N, 1)), "mass": np.ones(N), "fixed": np.zeros(N, bool),
         "vel": np.zeros((N, 3)), "omega": np.zeros((N, 3))}
    side = np.ceil(np.sqrt(sizes / 4.0)).astype(int)
    layers = -(-sizes // (side * side))
    half = np.ceil((side * CELL / 2.0 + 0.4) * 2.0) / 2.0
    height = np.ceil(layers * 2.2 + 1.0)
    t = 0.5
    for k, (sx, sy, sz, px, py, pz) in enumerate((
            (half, t, half, 0.0, -t, 0.0), (t, height / 2, half, half + t, height / 2, 0.0),
            (t, height / 2, half, -half - t, height / 2, 0.0), (half, height / 2, t, 0.0, height / 2, half + t),
            (half, height / 2, t, 0.0, height / 2, -half - t))):
        at = start[:-1] + k
        f["fixed"][at] = True
        for d, (s, p) in enumerate(((sx, px), (sy, py), (sz, pz))):
            f["scale"][at, d] = s
            f["pos"][at, d] = p
    # the heap's bodies
    n = int(sizes.sum())
    scene = np.repeat(np.arange(K), sizes)
    i = np.arange(n) - np.repeat(np.concatenate([[0], np.cumsum(sizes)[:-1]]), sizes)
    at = start[scene] + 5 + i
    column, layer = i % (side[scene] ** 2), i // (side[scene] ** 2)
    shape = rng.permutation(np.arange(n) % len(mesh))
    scale = 0.5 * (0.5 + np.floor(rng.random(n) * 77.0) / 128.0)
    yaw, lean, tilt = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, 2 * np.pi, n), rng.uniform(0.0, 0.004, n)
    zero = np.zeros(n)
    q = _qmul(np.stack([zero, np.sin(yaw / 2), zero, np.cos(yaw / 2)], -1), down[shape])
    q = _qmul(np.stack([np.cos(lean) * np.sin(tilt / 2), zero, np.sin(lean) * np.sin(tilt / 2), np.cos(tilt / 2)], -1), q)
    row = _matrix(q)[:, 1, :]
    low, high = np.zeros(n), np.zeros(n)
    for k in range(len(mesh)):
        m = shape == k
        y = (row[m] @ verts[k].T) * scale[m, None]
        low[m], high[m] = y.min(1), y.max(1)
    sink = rng.uniform(0.0, 0.004, n)
    y = np.zeros(n)
    top = np.zeros((K, int((side ** 2).max())))
    for k in range(int(layers.max())):
        m = layer == k
        y[m] = top[scene[m], column[m]] - low[m] - sink[m]
        top[scene[m], column[m]] = y[m] + high[m]
    x = (column % side[scene] + 0.5 - side[scene] / 2.0) * CELL + rng.uniform(-0.05, 0.05, n)
    z = (column // side[scene] + 0.5 - side[scene] / 2.0) * CELL + rng.uniform(-0.05, 0.05, n)
    speed = np.where(rng.random(n) < 0.1, 1.0, 0.1)   # a tenth of the bodies has just been dropped
    f["mesh"][at], f["scale"][at], f["pos"][at], f["rot"][at] = shape, scale[:, None], np.stack([x, y, z], -1), q
    f["mass"][at] = volume[shape] * scale ** 3
    f["vel"][at], f["omega"][at] = rng.normal(size=(n, 3)) * speed[:, None], rng.normal(size=(n, 3)) * 0.1
    cons = []
    for s in np.nonzero(links > 0)[0]:
        _hang(f, cons, rng, int(start[s] + 5 + sizes[s]), int(links[s]), JOINTS[int(rng.integers(0, 2))],
              float(height[s] + 0.6 * links[s] + 1.0))
    return _batch(f, cons, K, substeps)


def _hang(f, cons, rng, first, links, joint, y):
    """An anchor at height y (body `first`) and a chain of links below it."""
    q = S._axis_rotation(rng.normal(size=3)) if joint == "hinge" else (0.0, 0.0, 0.0, 1.0)
    turn = _matrix(np.asarray(q))
    down = turn @ np.array([0.0, -1.0, 0.0])
    at = slice(first, first + links + 1)
    f["rot"][at] = q
    f["scale"][at] = LINK
    f["scale"][first] = 0.1
    f["fixed"][first] = True
    f["mass"][at] = 8.0 * LINK[0] * LINK[1] * LINK[2]
    f["pos"][at] = np.array([0.0, y, 0.0]) + np.outer(np.concatenate([[0.0], 0.4 + 0.6 * np.arange(links)]), down)
    f["vel"][first + 1:first + links + 1] = rng.normal(0.0, 0.5, size=(links, 3))
    f["omega"][first + 1:first + links + 1] = rng.normal(0.0, 0.5, size=(links, 3))   # the chain is swinging
    for i in range(links):
        a, b, r1 = first + i, first + i + 1, (0.0, -0.1 if i == 0 else -0.3, 0.0)
        if joint == "hinge":
            cons.append(S.Constraint("hinge", a, b, r1, (0.0, 0.3, 0.0), 0.0, axis1=S.POS_X, axis2=S.POS_X, limited=True,
                                     limit_axis1=S.POS_Y, limit_axis2=S.POS_Y, lower=-0.5 * math.pi, upper=0.5 * math.pi))
        elif joint == "spherical":
            cons.append(S.Constraint("spherical", a, b, r1, (0.0, 0.3, 0.0), swing_axis1=S.POS_Y, swing_axis2=S.POS_Y,
                                     twist_axis1=S.POS_X, twist_axis2=S.POS_X, swing_lower=-math.pi, swing_upper=math.pi,
                                     twist_lower=-math.pi, twist_upper=math.pi))
        else:
            # a spring, as the reference's spring example joins its cube to its attachment
            cons.append(S.Constraint("positional", a, b, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 0.001,
                                     distance=tuple(-down * (0.3 if i == 0 else 0.5))))


def _batch(f, cons, scenes, substeps):
    N = len(f["mass"])
    return S.SceneBatch("batch", _Shapes.get()[0], f["scene"], f["mesh"], f["scale"], f["pos"], f["rot"], f["mass"], f["fixed"],
                        np.full(N, 0.5), np.full(N, 0.3), np.zeros(N), f["vel"], f["omega"], cons, num_scenes=scenes, dt=DT,
                        substeps=substeps, gravity=GRAVITY)


def _chains(scenes, links, seed, substeps, joints=JOINTS):
    """One chain per scene, of joint kind s modulo the kinds."""
    rng = np.random.default_rng(seed)
    N = scenes * (links + 1)
    f = {"scene": np.repeat(np.arange(scenes, dtype=np.int32), links + 1), "mesh": np.zeros(N, np.int32), "scale": np.zeros((N, 3)),
         "pos": np.zeros((N, 3)), "rot": np.zeros((N, 4)), "mass": np.ones(N), "fixed": np.zeros(N, bool),
         "vel": np.zeros((N, 3)), "omega": np.zeros((N, 3))}
    cons = []
    for s in range(scenes):
        _hang(f, cons, rng, s * (links + 1), links, joints[s % len(joints)], 0.6 * links + 1.0)
    return _batch(f, cons, scenes, substeps)


def _sphere_scenes(scenes, bodies, seed, substeps):
    """Spheres dropped in a column with a compound body of two boxes on top, touching from the start."""
    out = []
    rng = np.random.default_rng(seed)
    for _ in range(scenes):
        b = S._Builder("spheres")
        S._floor(b, (6.0, 0.5, 6.0))
        y = 0.0
        for _ in range(bodies):
            r = float(np.float32(rng.uniform(0.3, 0.6)))
            b.body([S.Collider("sphere", radius=r)], (float(rng.uniform(-0.05, 0.05)), y + r - 0.002, float(rng.uniform(-0.05, 0.05))),
                   mass=1.0, v=tuple(rng.normal(0, 0.3, size=3)))
            y += 2.0 * r - 0.006
        cube = b.mesh("cube")
        b.body([S.Collider("hull", cube, (0.3, 0.3, 0.3)), S.Collider("hull", cube, (0.6, 0.1, 0.1))], (0.1, y + 0.297, 0.05),
               mass=2.0)
        out.append(b.finish(dt=DT, substeps=substeps))
    return out


# -- one case ---------------------------------------------------------------------------------------
def _scene_batch(case, seed):
    """The case's scenes as one batch (every kind but the spheres), made from the seed alone."""
    kind = case["kind"]
    if kind == "stack":
        s = S.stack_scene(case["bodies"], seed)
        n = s.num_bodies
        scale = np.array([c[0].scale for c in s.colliders])
        return S.SceneBatch("stack", s.meshes, np.zeros(n, np.int32), np.zeros(n, np.int32), scale, s.pos, s.rot, s.mass, s.fixed,
                            s.mus, s.mud, s.rest, s.vel, s.omega, substeps=case["substeps"])
    if kind == "towers":
        return S.tower_batch(case["scenes"], case["bodies"], seed=seed, substeps=case["substeps"])
    if kind in ("heap", "queries"):
        return _heaps([case["bodies"]], [0], seed, case.get("substeps", 20))
    if kind == "batch":
        # sizes are spread evenly over their log-uniform range and links over theirs, in an order that
        # depends on the case alone: every seed gives states of one shape
        rng, n = np.random.default_rng(7), case["scenes"]
        even = (np.arange(n) + 0.5) / n
        sizes = np.exp(rng.permutation(even) * math.log((case["most"] + 1) / 2.0) + math.log(2.0)).astype(int)
        links = np.where(rng.permutation(even) < 0.25, (8 + 57 * rng.permutation(even)).astype(int), 0)
        return _heaps(sizes, links, seed, case["substeps"])
    if kind == "chains":
        return _chains(case["scenes"], case["links"], seed, case["substeps"])
    return _chains(case["scenes"], case["links"], seed, case["substeps"], JOINTS[:2])  # swing


def prepare(case, seed):
    kind = case["kind"]
    w = rawphys.World(0, case.get("precision", "fp64"))   # the gradients are FP64
    st = {"kind": kind, "world": w, "collisions": kind != "chains"}
    if kind == "spheres":
        scenes = _sphere_scenes(case["scenes"], case["bodies"], seed, case["substeps"])
        for k, s in enumerate(scenes):
            w.load(s, 0 if k == 0 else w.new_scene())
        st["substeps"] = case["substeps"]
    elif kind == "dominoes":
        batch, last, target = S.domino_batch(case["scenes"], seed, case["bodies"], case["bodies"])
        batch.substeps = case["substeps"]
        w.load_batch(batch)
        st.update(last=last, target=target, frames=case["frames"])
    else:
        batch = _scene_batch(case, seed)
        w.load_batch(batch)
        st["substeps"] = batch.substeps
        if kind == "swing":
            n = case["links"] + 1
            last = n * np.arange(case["scenes"], dtype=np.int32) + case["links"]
            target = batch.pos[last] + np.random.default_rng([seed, 3]).normal(0.0, 0.3, size=(case["scenes"], 3))
            st.update(last=last, target=target, frames=case["frames"], collisions=False)
    if "last" not in st:
        st["start"] = w.get_state()
        st["out"] = np.empty_like(st["start"])
        if kind == "queries":   # the caller's pair buffer, as rp_broad_pairs takes one
            st["pairs"] = np.zeros((8 * len(st["start"]), 2), dtype=np.int32)
    return st


def run(state):
    w = state["world"]
    if "last" in state:
        return w.adjoint(state["frames"], state["last"], state["target"], checkpoint_every=10, collisions=state["collisions"])
    w.set_state(state["start"])
    if state["kind"] == "queries":
        vertices, normals = w.transformed_hulls()
        found, pairs = w.broad_pairs(0), state["pairs"]
        pairs[:len(found)] = found
        return {"pairs": pairs, "vertices": vertices, "normals": normals}
    w.simulate(DT, state["substeps"], 1, state["collisions"], 1)
    return w.get_state(state["out"])


def _counts(case):
    """(bodies, dynamic bodies, joints, mean hull vertices) of a case; a batch's sizes are log-uniform."""
    kind = case["kind"]
    if kind == "batch":
        mean = (case["most"] - 1) / math.log((case["most"] + 1) / 2.0)
        return case["scenes"] * (mean + 5 + 9.25), case["scenes"] * (mean + 9), case["scenes"] * 9, 31
    if kind in ("chains", "swing"):
        return case["scenes"] * (case["links"] + 1), case["scenes"] * case["links"], case["scenes"] * case["links"], 8
    scenes = case.get("scenes", 1)
    fixed = 5 if kind in ("heap", "queries") else 1
    return scenes * (case["bodies"] + fixed + 1), scenes * case["bodies"], 0, 31 if fixed == 5 else 8


def work(case):
    """Bytes: the state records read and written (2 x 224 B), masses, inertia and material (about 80 B) once
    a body; a query writes its vertices, normals and pairs. Flops a substep: predict and velocity update
    about 400 a body; two resting contacts' share of GJK, EPA, clipping and the two solves about 6000 a
    body where bodies collide; about 1500 a joint; a gradient is about four forward passes."""
    bodies, dynamic, joints, verts = _counts(case)
    if case["kind"] == "queries":
        return {"bytes": bodies * (64 + verts * 24 * 3 + 60), "flops": bodies * verts * 18 * 3}
    touch = case["kind"] not in ("chains", "swing")
    flops = case["substeps"] * case.get("frames", 1) * (dynamic * (400 + 6000 * touch) + joints * 1500)
    if case["kind"] in ("dominoes", "swing"):
        return {"bytes": bodies * (224 + 80 + 72), "flops": 4 * flops}
    return {"bytes": bodies * (448 + 80), "flops": flops}


# -- the same numbers in 64 bits ------------------------------------------------------------------
def exact(case, seed):
    """What run() returns, in plain numpy at 64 bits: the joint chains' step and the transformed hulls.
    Scenes with contacts have none (a serial GJK, EPA and clipping of each pair of every substep in plain
    numpy takes minutes at these sizes), nor have the gradients, which are derivatives of such steps."""
    if case["kind"] == "queries":
        b = _scene_batch(case, seed)
        out, norms = [None] * b.num_bodies, [None] * b.num_bodies
        turn = _matrix(b.rot)
        for k, (vert, norm) in enumerate(_hull_tables()):
            for i in np.nonzero(b.mesh == k)[0]:
                out[i] = (vert * b.scale[i]) @ turn[i].T + b.pos[i]
                m = norm / b.scale[i]
                norms[i] = (m / np.linalg.norm(m, axis=1, keepdims=True)) @ turn[i].T
        return {"normals": np.concatenate(norms), "pairs": None, "vertices": np.concatenate(out)}
    if case["kind"] != "chains" or case["scenes"] * case["links"] * case["substeps"] > 768 * 64 * 25:
        return None
    return _exact_chains(_scene_batch(case, seed), case["scenes"], case["links"], case["substeps"])


def _hull_tables():
    """Per mesh: hull vertices in order of first use and one outward normal per planar face in order of its
    first triangle (the order the hull builder keeps)."""
    for m in _Shapes.get()[0]:
        p = m.positions.astype(np.float64)
        _, first = np.unique(p, axis=0, return_index=True)
        tri = p.reshape(-1, 3, 3)
        n = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        keep = []
        for i in range(len(n)):
            if not any(np.dot(n[i], n[j]) > 1 - 1e-6 for j in keep):
                keep.append(i)
        yield p[np.sort(first)], n[keep]


def _cross(a, b):
    return np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                     a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], -1)


def _dot(a, b):
    return np.sum(a * b, -1)


def _unit(v):
    n = np.linalg.norm(v, axis=-1, keepdims=True)
    return v / np.where(n > 0, n, 1.0), n[..., 0]


class _Link:
    """Link i of every chain of one joint kind, as the solver sees it."""

    def __init__(self, c, i):
        self.c, self.i = c, i
        self.q = c["q"][:, i]
        self.turn = _matrix(self.q)
        self.inertia = self.turn * c["Ii"][:, i][:, None, :] @ np.swapaxes(self.turn, -1, -2)
        self.invm = c["invm"][:, i]
        self.moves = c["invm"][0, i] > 0

    def axis(self, k):
        return self.turn[:, :, k]

    def rotate(self, turn, sign):
        """q <- normalised q + sign / 2 (turn, 0) q."""
        if self.moves:
            d = _qmul(np.concatenate([turn, np.zeros((len(turn), 1))], -1), self.q)
            self.c["q"][:, self.i] = _unit(self.q + 0.5 * sign * d)[0]


def _apply(a):
    return lambda v: np.einsum("sij,sj->si", a.inertia, v)


def _positional(c, i, j, r1, r2, compliance, h, gap):
    """One positional correction between links i and j (the multiplier starts at zero every substep)."""
    a, b = _Link(c, i), _Link(c, j)
    ra, rb = np.einsum("sij,j->si", a.turn, r1), np.einsum("sij,j->si", b.turn, r2)
    dx = gap(ra, rb)
    n, size = _unit(dx)
    wa = a.invm + _dot(_cross(ra, n), _apply(a)(_cross(ra, n)))
    wb = b.invm + _dot(_cross(rb, n), _apply(b)(_cross(rb, n)))
    impulse = (-size / (wa + wb + compliance / (h * h)))[:, None] * n
    c["x"][:, i] += a.invm[:, None] * impulse
    c["x"][:, j] -= b.invm[:, None] * impulse
    a.rotate(_apply(a)(_cross(ra, impulse)), 1.0)
    b.rotate(_apply(b)(_cross(rb, impulse)), -1.0)


def _angular(c, i, j, turn, where):
    a, b = _Link(c, i), _Link(c, j)
    n, size = _unit(turn)
    w = _dot(n, _apply(a)(n)) + _dot(n, _apply(b)(n))
    impulse = np.where(where & (size > 0), size / w, 0.0)[:, None] * n
    a.rotate(_apply(a)(impulse), 1.0)
    b.rotate(_apply(b)(impulse), -1.0)


def _hinge_limit(c, i, j, lo, hi):
    a, b = _Link(c, i), _Link(c, j)
    n, n1, n2 = a.axis(0), a.axis(1), b.axis(1)
    phi = np.arcsin(np.clip(_dot(_cross(n1, n2), n), -1.0, 1.0))
    phi = np.where(_dot(n1, n2) < 0.0, np.pi - phi, phi)
    phi = np.where(phi > np.pi, phi - 2 * np.pi, phi)
    where = (phi < lo) | (phi > hi)
    half = 0.5 * np.clip(phi, lo, hi)
    q = np.concatenate([n * np.sin(half)[:, None], np.cos(half)[:, None]], -1)
    _angular(c, i, j, _cross(np.einsum("sij,sj->si", _matrix(q), n1), n2), where)


def _exact_chains(b, scenes, links, substeps):
    n, h = links + 1, DT / substeps
    shape = (scenes, n)
    x, q = b.pos.reshape(shape + (3,)).copy(), b.rot.reshape(shape + (4,)).copy()
    v, w = b.vel.reshape(shape + (3,)).copy(), b.omega.reshape(shape + (3,)).copy()
    moves = ~b.fixed.reshape(shape)
    sq = b.scale.reshape(shape + (3,)) ** 2
    I = b.mass.reshape(shape)[..., None] * np.stack([sq[..., 1] + sq[..., 2], sq[..., 0] + sq[..., 2], sq[..., 0] + sq[..., 1]], -1)
    Ii, invm = np.where(moves[..., None], 1.0 / I, 0.0), np.where(moves, 1.0 / b.mass.reshape(shape), 0.0)
    still = (np.linalg.norm(v, axis=-1) < 0.1) & (np.linalg.norm(w, axis=-1) < 0.1) & moves
    rest = np.where(still, DT, 0.0)
    distance = np.array([con.distance for con in b.constraints]).reshape(scenes, links, 3)
    px, pq, pv, pw = x.copy(), q.copy(), v.copy(), w.copy()
    mv = moves[..., None]
    for _ in range(substeps):
        px, pq = x.copy(), q.copy()
        v = np.where(mv, v + h * np.array([0.0, -GRAVITY, 0.0]), v)
        x = x + h * np.where(mv, v, 0.0)
        turn = _matrix(q)
        local = np.einsum("snji,snj->sni", turn, w)
        spin = np.cross(w, np.einsum("snij,snj->sni", turn, I * local))
        w = np.where(mv, w - h * np.einsum("snij,snj->sni", turn, Ii * np.einsum("snji,snj->sni", turn, spin)), w)
        dq = _qmul(np.concatenate([w, np.zeros(shape + (1,))], -1), q)
        q = np.where(mv, _unit(q + 0.5 * h * dq)[0], q)
        for k in range(3):
            part = slice(k, scenes, 3)
            if k >= scenes:
                continue
            c = {"x": x[part].copy(), "q": q[part].copy(), "Ii": Ii[part], "invm": invm[part]}
            for i in range(links):
                r1, r2 = np.array([0.0, -0.1 if i == 0 else -0.3, 0.0]), np.array([0.0, 0.3, 0.0])
                if k == 2:
                    zero = np.zeros(3)
                    _positional(c, i, i + 1, zero, zero, 0.001, h,
                                lambda ra, rb: c["x"][:, i] - c["x"][:, i + 1] - distance[part, i])
                    continue
                if k == 0:
                    # the aligned axes first: the correction turns a's axis onto b's
                    _angular(c, i, i + 1, _cross(_Link(c, i).axis(0), _Link(c, i + 1).axis(0)), True)
                _positional(c, i, i + 1, r1, r2, 0.0, h, lambda ra, rb: c["x"][:, i] + ra - c["x"][:, i + 1] - rb)
                if k == 0:
                    _hinge_limit(c, i, i + 1, -0.5 * math.pi, 0.5 * math.pi)
            x[part], q[part] = c["x"], c["q"]
        pv, pw = np.where(mv, v, pv), np.where(mv, w, pw)
        v = np.where(mv, (x - px) / h, v)
        dq = _qmul(q, pq * np.array([-1.0, -1.0, -1.0, 1.0]))
        w = np.where(mv, 2.0 / h * np.where(dq[..., 3:] >= 0.0, 1.0, -1.0) * dq[..., :3], w)
    one = np.ones(shape + (1,))
    return np.concatenate([x, q, v, w, px, pq, pv, pw, one, rest[..., None]], -1).reshape(scenes * n, 28)
