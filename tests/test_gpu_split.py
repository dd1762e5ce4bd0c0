"""Work split over lanes, blocks and workers, at the sizes where a split changes: the FP64 solves' eight lanes
a node, the grid sweeps without level barriers, the sorted broad phase's pieces, the narrow solve blocks and
the adjoint's workers. FP64 results equal the oracle's bit for bit."""
import math

import numpy as np
import pytest

import rawphys
from oracle.oracle import Oracle
from rawphys import scenes as S

pytestmark = pytest.mark.gpu


def _joint_scene(axis, other):
    # links in free fall joined by every joint type along one pair of body axes, limits acting on both sides
    b = S._Builder("axes%d%d" % (axis, other))
    rng = np.random.default_rng(10 * axis + other)
    for i in range(6):
        q = rng.normal(size=4)
        b.hull_body("cube", (0.1, 0.3, 0.2), (0.0, -0.6 * i, 0.0), rot=tuple(q / np.linalg.norm(q)), mass=0.5 + i, fixed=i == 0,
                    v=tuple(rng.normal(size=3)), w=tuple(rng.normal(size=3)))
    r1, r2 = (0.0, -0.3, 0.05), (0.02, 0.3, 0.0)
    b.scene.constraints += [
        S.Constraint("hinge", 0, 1, r1, r2, 0.0, axis1=axis, axis2=axis, limited=True, limit_axis1=other, limit_axis2=other,
                     lower=-0.2, upper=0.3),
        S.Constraint("spherical", 1, 2, r1, r2, swing_axis1=axis, swing_axis2=other, twist_axis1=other, twist_axis2=axis,
                     swing_lower=-0.4, swing_upper=0.2, twist_lower=-0.1, twist_upper=0.5),
        S.Constraint("mutual_orientation", 2, 3, compliance=1e-5),
        S.Constraint("positional", 3, 4, r1, r2, 1e-4, distance=(0.1, 0.4, 0.0)),
        S.Constraint("hinge", 4, 5, r1, r2, 1e-6, axis1=axis, axis2=other),
    ]
    return b.finish(dt=1.0 / 60.0, substeps=10, pos_iters=1, collisions=False, steps=1)


@pytest.mark.parametrize("axis,other", [(0, 2), (1, 4), (2, 5), (3, 0), (4, 1), (5, 3)])
def test_eight_lane_joint_solves_equal_the_oracle(axis, other):
    sc = _joint_scene(axis, other)
    o = Oracle("port").load(sc)
    o.step(4)
    for extra in (0, 641):      # with a large scene beside it the world takes the sweep kernels
        w = rawphys.World(0, "fp64")
        w.load(sc)
        if extra:
            w.load(S.stack_scene(extra, seed=1), w.new_scene())
        w.simulate(sc.dt, sc.substeps, 1, False, 4)
        assert np.array_equal(w.get_state()[:sc.num_bodies], o.get_state()), extra
        w.close()


@pytest.mark.parametrize("bodies,iters,mode", [(700, 1, "phased"), (700, 2, "persistent"), (1400, 2, "phased")])
def test_grid_sweeps_without_level_barriers_equal_the_oracle(bodies, iters, mode):
    # one settling pile: levels from one node to hundreds, pairs of up to 32 contacts
    sc = S.large_scene(bodies, seed=bodies)
    w = rawphys.World(0, "fp64")
    w.set_mode(mode)
    w.load(sc)
    w.step(45)
    start = w.get_state()
    w.simulate(sc.dt, 5, iters, True, 1)
    o = Oracle("port").load(sc)
    o.set_state(start)
    o.step(1, substeps=5, pos_iters=iters)
    assert np.array_equal(w.get_state(), o.get_state())
    w.close()


def _spread(n, seed):
    # a band of bodies whose x intervals all overlap (longer than a warp's piece of 1024), wide bodies that reach
    # every other one, and pairs at the exact distance of the test and one step beyond it
    rng = np.random.default_rng(seed)
    b = S._Builder("spread%d" % n)
    b.hull_body("cube", (30.0, 0.5, 30.0), (0.0, -0.5, 0.0), fixed=True)
    r = math.sqrt(3.0 * 0.2 * 0.2)
    for i in range((n - 1) // 2):
        p = (rng.uniform(-0.2, 0.2), rng.uniform(0.0, 40.0), rng.uniform(-40.0, 40.0))
        d = 2.0 * r + 0.1
        if i % 2:
            d = np.nextafter(d, 10.0)
        b.hull_body("cube", (0.2, 0.2, 0.2), p, mass=1.0)
        b.hull_body("cube", (0.2, 0.2, 0.2), (p[0], p[1], p[2] + d), mass=1.0)
    while len(b._pos) < n:
        b.hull_body("cube", (3.0, 0.1, 0.1), tuple(rng.uniform(-5.0, 5.0, size=3)), mass=1.0)
    return b.finish(dt=1.0 / 60.0, substeps=2, pos_iters=1, collisions=True, steps=1)


@pytest.mark.parametrize("n", [1024, 1026, 2048, 2049, 4000])
def test_sorted_broad_phase_equals_the_oracle(n):
    sc = _spread(n, seed=n)
    ref = Oracle("port").load(sc).broad_pairs()
    for precision in ("fp64", "fp32"):
        w = rawphys.World(0, precision)
        w.load(sc)
        assert np.array_equal(w.broad_pairs(), ref), precision
        w.close()


def test_sorted_broad_phase_overflow_regrows(monkeypatch):
    # 5140 pairs; scratch of 16 pairs a body times the scale holds 1204, then 4816, then 19264
    sc = S.large_scene(1500, seed=4)
    states = []
    for scale in (None, "0.05"):
        if scale:
            monkeypatch.setenv("RP_SCRATCH_SCALE", scale)
        w = rawphys.World(0, "fp64")
        w.load(sc)
        w.simulate(sc.dt, 2, 1, True, 2)
        states.append(w.get_state())
        w.close()
    assert np.array_equal(*states)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_many_small_scenes_equal_few(precision):
    # more small scenes than the device holds blocks of 128 threads: 64 threads each, the same bits
    scs = [S.stack_scene(n, seed=n) for n in (3, 30)] + [S.chain_scene(5, "hinge", seed=2)]
    states = []
    for copies in (1, 320):
        w = rawphys.World(0, precision)
        first = [w.load(sc, 0 if (c, k) == (0, 0) else w.new_scene()) for c in range(copies) for k, sc in enumerate(scs)]
        w.simulate(1.0 / 60.0, 10, 1, True, 2)
        state = w.get_state()
        states.append([[state[f:f + sc.num_bodies] for f, sc in zip(first[c * 3:], scs)] for c in (0, copies - 1)])
        w.close()
    for got in states[1]:
        for a, b in zip(states[0][0], got):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_one_pass_contacts_equal_separate_kernels(precision):
    # a small world takes EPA and manifold in one kernel with GJK, one of more pair slots (16 a body) than 48 a
    # resident warp, 116736, apart
    piles = [S.random_pile_scene(n, seed=n) for n in (2, 9, 20)] + [S.tower_scene(8, seed=1), S.chain_scene(6, "spherical", seed=3)]
    others = [S.random_pile_scene(24, seed=k % 8) for k in range(400)]
    states = []
    for scs in (piles, piles + others):
        w = rawphys.World(0, precision)
        first = [w.load(sc, 0 if k == 0 else w.new_scene()) for k, sc in enumerate(scs)]
        w.simulate(1.0 / 60.0, 20, 1, True, 40)
        state = w.get_state()
        states.append([state[f:f + sc.num_bodies] for f, sc in zip(first, piles)])
        w.close()
    for sc, a, b in zip(piles, *states):
        assert np.array_equal(a, b), sc.name


def test_adjoint_in_groups_equals_all_at_once():
    # 64 scenes tape a few substeps at a time, one scene all of its segment's: the same gradients, bit for bit
    batch, last, target = S.domino_batch(64, seed=2, min_dominoes=1, max_dominoes=3)
    w = rawphys.World(0, "fp64")
    w.load_batch(batch)
    res = w.adjoint(2, last, target, checkpoint_every=2, substeps=20)
    w.close()
    for s in (0, 31, 63):
        idx = np.nonzero(batch.scene == s)[0]
        w = rawphys.World(0, "fp64")
        w.load(S.batch_scene(batch, s))
        one = w.adjoint(2, [int(last[s]) - int(idx[0])], target[s], checkpoint_every=1 + s % 2, substeps=20)
        w.close()
        assert res["loss"][s] == one["loss"][0]
        for k in ("grad_v", "grad_w", "grad_mass", "grad_friction"):
            assert np.array_equal(res[k][idx], one[k]), (s, k)


def test_adjoint_of_a_wide_row_matches_central_differences():
    # 48 dominoes: levels of thousands of entries (beyond a chunk), children far beyond the ring
    sc = S.domino_scene(48, seed=1)
    n, h, substeps = sc.num_bodies, 1e-6, 3
    target = np.array([1.0, 1.5, 0.2])
    w = rawphys.World(0, "fp64")
    w.load(sc)
    start = w.get_state()
    res = w.adjoint(1, [n - 1], target, substeps=substeps)
    checks = []
    for col in (7, 8, 9, 10, 12):
        loss = []
        for sign in (1.0, -1.0):
            st = start.copy()
            st[n - 1, col] += sign * h
            w.set_state(st)
            w.simulate(sc.dt, substeps, sc.pos_iters, True, 1)
            loss.append(float(np.sum((w.get_state()[n - 1, 0:3] - target) ** 2)))
        checks.append(((loss[0] - loss[1]) / (2 * h), (res["grad_v"] if col < 10 else res["grad_w"])[n - 1, (col - 7) % 3]))
    w.close()
    scale = max(abs(fd) for fd, _ in checks)
    for fd, ad in checks:
        assert abs(ad - fd) <= 1e-3 * max(abs(fd), 1e-3 * scale), checks
