"""The solver's schedules from one substep, frame and launch form to the next: the level tables a substep
leaves behind and the ones the next starts from. FP64 results equal the oracle's bit for bit."""
import numpy as np
import pytest

import rawphys
from oracle.oracle import Oracle
from rawphys import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["phased", "persistent"])
def test_position_and_velocity_schedules_side_by_side(mode):
    # a single scene of 256 bodies or more: two CTAs build a substep's two schedules at the same time, 200 times
    # here; a velocity schedule without levels would leave out the whole velocity sweep
    sc = S.large_scene(300, seed=11)
    w = rawphys.World(0, "fp64")
    w.set_mode(mode)
    w.load(sc)
    w.step(150)
    o = Oracle("port").load(sc)
    o.set_state(w.get_state())
    for frame in range(10):
        w.simulate(sc.dt, 20, 1, True, 1)
        o.step(1, substeps=20)
        assert np.array_equal(w.get_state(), o.get_state()), frame
        for which in (0, 1):
            lev, bodies = w.last_schedule(which=which)
            # a node is one level above the latest of its bodies, in constraint order
            top, want = {}, []
            for l, pair in zip(lev, bodies):
                ends = [b for b in pair if b >= 0] if l >= 0 else []
                at = max([top.get(b, 0) for b in ends], default=-1)
                want.append(at)
                top.update((b, at + 1) for b in ends)
            assert np.array_equal(lev, want) and (lev >= 0).any(), (frame, which)
    w.close()


def _knot(n, seed):
    # n cubes around one point, every pair overlapping: n (n - 1) / 2 pairs with contacts, beyond the
    # 2 bodies + 32 nodes a scene-resident solve has room for when n > 6, in at least n - 1 levels
    rng = np.random.default_rng(seed)
    b = S._Builder("knot%d" % n)
    for _ in range(n):
        q = rng.normal(size=4)
        b.hull_body("cube", (0.5, 0.5, 0.5), tuple(rng.uniform(-0.3, 0.3, size=3)), rot=tuple(q / np.linalg.norm(q)), mass=1.0)
    return b.finish(dt=1.0 / 60.0, substeps=2, pos_iters=1, collisions=True, steps=1)


@pytest.mark.parametrize("substeps", [1, 2])
@pytest.mark.parametrize("modes", [("phased",) * 5, ("persistent", "phased", "persistent", "phased", "persistent")])
def test_deep_schedules_after_shallow_ones(modes, substeps):
    # A frame of deep schedules, one of a single level (with two substeps the first already ends shallow: the knot
    # bursts), a deep one again: what a shallow schedule leaves in the level tables must not keep a deeper one's
    # entries. Two scenes, so that the first one's tables and nodes end at the second's.
    scs = [_knot(24, 3), _knot(30, 4)]
    w = rawphys.World(0, "fp64")
    first = [w.load(sc, 0 if k == 0 else w.new_scene()) for k, sc in enumerate(scs)]
    tight = w.get_state()
    apart = tight.copy()
    for f, sc in zip(first, scs):
        n = sc.num_bodies   # pairs of touching cubes: one level
        apart[f:f + n, 0:3] = [(0.9 * (i % 2), 0.0, 4.0 * (i // 2)) for i in range(n)]
        apart[f:f + n, 3:7] = (0.0, 0.0, 0.0, 1.0)
    for i, mode in enumerate(modes):
        start = apart if i % 2 else tight
        w.set_mode(mode)
        w.set_state(start)
        w.simulate(1.0 / 60.0, substeps, 1, True, 1)
        got = w.get_state()
        for s, (f, sc) in enumerate(zip(first, scs)):
            n = sc.num_bodies
            for which in (0, 1) if substeps == 1 else ():
                lev, _ = w.last_schedule(s, which)
                if i % 2:
                    assert lev.max() == 0 and (lev >= 0).sum() == n // 2, (i, s, which)
                else:
                    assert lev.max() >= n - 2 and (lev >= 0).sum() == n * (n - 1) // 2, (i, s, which)
            o = Oracle("port").load(sc)
            o.set_state(start[f:f + n])
            o.step(1, substeps=substeps)
            assert np.array_equal(got[f:f + n], o.get_state()), (i, s)
    w.close()
