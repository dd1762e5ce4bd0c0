"""Hulls at the edges of the narrowphase's topology records and clip storage (96 planes): faces with more neighbours
than planes are kept, and topologies made by the caller."""
import ctypes as C

import numpy as np
import pytest

import rawphys
from oracle.oracle import Oracle
from rawphys import meshes as M
from rawphys import scenes as S

pytestmark = pytest.mark.gpu

CLIP_OVERFLOW = 1 << 3
# FP32 against FP64: which contact points act is decided by roundings here, so the forms may differ by what the
# contacts move in two frames: the 2 mm of penetration and the fall, g t^2 / 2 = 5.6 mm
NEAR = 8e-3


def _wedge(arc):
    # two apexes joined by an edge and `arc` points on a circle around it: arc + 2 vertices, 2 arc faces, and the
    # two faces on the edge share a vertex with every other one: 2 arc - 1 neighbours
    t = np.linspace(-1.2, 1.2, arc)
    p = np.stack([np.cos(t), np.sin(t), 0.0 * t], axis=1) - np.array([0.4, 0.0, 0.0])
    top, bottom = np.array([-0.4, 0.0, 1.0]), np.array([-0.4, 0.0, -1.0])
    tris = [[apex, p[i], p[i + 1]] for i in range(arc - 1) for apex in (top, bottom)]
    tris += [[top, bottom, p[0]], [top, bottom, p[-1]]]
    return M.Mesh("wedge%d" % arc, M._orient_outward(np.asarray(tris)))


def _face_to_face(arc):
    # a fixed wedge with an edge face up and one lying on it, 2 mm deep: whichever face is the reference, it
    # has all the other faces as neighbours
    b = S._Builder("wedges%d" % arc)
    b.scene.meshes.append(_wedge(arc))
    wedge = [S.Collider("hull", 0, (1.0, 1.0, 1.0))]
    h = 0.4 * np.sin(1.2)   # of the edge above the origin once the face is level
    b.body(wedge, (0.0, 0.0, 0.0), rot=(0.0, 0.0, -np.sin(0.6), np.cos(0.6)), fixed=True)
    b.body(wedge, (0.05, 2.0 * h - 0.002, 0.03), rot=(0.0, 0.0, np.sin(0.6), np.cos(0.6)), mass=1.0)
    return b.finish(dt=1.0 / 60.0, substeps=10, pos_iters=1, collisions=True, steps=1)


def _run(sc, precision="fp64", mode="phased", frames=2, hulls=None):
    w = rawphys.World(0, precision)
    w.set_mode(mode)
    if hulls:
        w._hulls.update(hulls(w, sc))
    w.load(sc)
    w.step(frames)
    out = w.get_state(), w.status(), len(w.last_contacts()[0])
    w.close()
    return out


def _oracle(sc, frames=2):
    o = Oracle("port").load(sc)
    o.step(frames)
    assert o.error_bits() == 0
    return o.get_state()


def test_a_face_with_95_neighbours_equals_the_oracle():
    sc = _face_to_face(48)
    state, status, contacts = _run(sc)
    assert status == 0 and contacts >= 1
    assert np.array_equal(state, _oracle(sc))
    single, status, contacts = _run(sc, "fp32")
    assert status == 0 and contacts >= 1
    assert np.abs(single[:, 0:7] - state[:, 0:7]).max() <= NEAR


@pytest.mark.parametrize("arc", [49, 62])
def test_a_face_with_more_neighbours_than_planes_reports_it(arc):
    # 97 and 123 neighbours: 96 planes are kept and the status says so, in every form
    sc = _face_to_face(arc)
    states = []
    for precision, mode in (("fp64", "phased"), ("fp64", "persistent"), ("fp32", "phased"), ("fp32", "persistent")):
        state, status, contacts = _run(sc, precision, mode)
        assert status == CLIP_OVERFLOW and contacts >= 1, (precision, mode)
        states.append(state)
    assert np.array_equal(states[0], states[1])
    for single in states[2:]:
        assert np.abs(single[:, 0:7] - states[0][:, 0:7]).max() <= NEAR


def _two_cubes():
    b = S._Builder("two")
    b.hull_body("cube", (0.5, 0.5, 0.5), (0.0, 0.0, 0.0), fixed=True)
    b.hull_body("cube", (0.5, 0.5, 0.5), (0.1, 0.998, 0.05), mass=1.0)
    return b.finish(dt=1.0 / 60.0, substeps=10, pos_iters=1, collisions=True, steps=1)


def _from_topology(change):
    # the scene's cube through the caller's own topology tables, changed by `change`
    def hulls(w, sc):
        m = sc.meshes[0]
        v, n, t = w.hull_topology(w.hull(m.positions.astype(np.float64) * 0.5, m.indices))
        rows = {k: [list(data[start[i]:start[i + 1]]) for i in range(len(start) - 1)] for k, (start, data) in t.items()}
        n = change(rows, n)
        args = []
        for k in range(4):
            args.append(np.concatenate([[0], np.cumsum([len(r) for r in rows[k]])]).astype(np.int32))
            args.append(np.array([x for r in rows[k] for x in r], dtype=np.int32))
        v, n = np.ascontiguousarray(v), np.ascontiguousarray(n)
        out = C.c_int()
        ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double if a.dtype == np.float64 else C.c_int))
        w._check(w.lib.rp_hull_create_from_topology(w.h, ptr(v), len(v), ptr(n), len(n), *[ptr(a) for a in args], C.byref(out)))
        return {(id(m), (0.5, 0.5, 0.5)): out.value}
    return hulls


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_repeated_neighbours_of_a_callers_topology_report_the_overflow(precision):
    # every neighbour 25 times over: 100 planes, in the phased form's warp kernels and the persistent form's
    # general code
    def repeat(rows, n):
        rows[3] = [r * 25 for r in rows[3]]
        return n
    sc = _two_cubes()
    states = []
    for mode in ("phased", "persistent"):
        state, status, contacts = _run(sc, precision, mode, hulls=_from_topology(repeat))
        assert status == CLIP_OVERFLOW and contacts >= 1, mode
        states.append(state)
    if precision == "fp64":
        assert np.array_equal(*states)
    assert np.abs(states[0][:, 0:7] - states[1][:, 0:7]).max() <= NEAR


def test_a_callers_topology_with_an_empty_face():
    def empty_face(rows, n):
        rows[0].append([])
        rows[3].append([])
        return np.vstack([n, [[0.0, 0.0, 1.0]]])
    sc = _two_cubes()
    plain = _run(sc)
    state, status, contacts = _run(sc, hulls=_from_topology(empty_face))
    assert status == 0 and contacts == plain[2]
    assert np.array_equal(state, plain[0])


def test_a_vertex_of_no_triangle():
    sc = _two_cubes()
    m = M.cube()
    m.positions = np.ascontiguousarray(np.vstack([m.positions, [[0.25, 0.5, 0.125]]]), dtype=np.float32)
    sc.meshes[0] = m
    state, status, contacts = _run(sc)
    assert status == 0 and contacts >= 1
    assert np.array_equal(state, _oracle(sc))
