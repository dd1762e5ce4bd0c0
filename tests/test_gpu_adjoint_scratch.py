"""The adjoint's tapes: scenes without anything to differentiate, and how much scratch a call takes."""
import numpy as np
import pytest

import rawphys
from rawphys import scenes as S

pytestmark = pytest.mark.gpu
KEYS = ("grad_v", "grad_w", "grad_mass", "grad_friction")


@pytest.mark.parametrize("collisions", [True, False])
def test_a_scene_of_fixed_bodies_in_a_batch(collisions):
    # its tape holds inputs only; the scenes beside it are what they are without it
    batch, last, target = S.domino_batch(3, seed=5, min_dominoes=1, max_dominoes=2)
    floor = S._Builder("floor")
    S._floor(floor)
    floor.hull_body("cube", (0.5, 0.5, 0.5), (0.0, 0.4, 0.0), fixed=True)
    floor = floor.finish(dt=1.0 / 60.0, substeps=20, pos_iters=1, collisions=True, steps=1)
    w = rawphys.World(0, "fp64")
    w.load_batch(batch)
    alone = w.adjoint(2, last, target, substeps=5, collisions=collisions)
    w.close()
    w = rawphys.World(0, "fp64")
    n = w.load_batch(batch) + batch.num_bodies
    f = w.load(floor, w.new_scene())
    assert f == n
    res = w.adjoint(2, [int(e) for e in last] + [f + 1], np.vstack([target, [[1.0, 2.0, 3.0]]]), substeps=5, collisions=collisions)
    w.close()
    assert np.array_equal(res["loss"][:3], alone["loss"])
    assert res["loss"][3] == 1.0 + 1.6 ** 2 + 9.0
    for k in KEYS:
        assert np.array_equal(res[k][:n], alone[k]), k
        assert not np.any(res[k][n:]), k


def test_scenes_take_turns_where_their_tapes_do_not_fit(monkeypatch):
    # the same gradients from one substep of one scene at a time (1 byte of room), from a few scenes at a time and
    # from all at once; the launches tell how many turns there were
    batch, last, target = S.domino_batch(6, seed=9, min_dominoes=1, max_dominoes=4)
    results, launches = [], []
    for room in (None, "1", str(20 << 20)):
        if room:
            monkeypatch.setenv("RP_ADJOINT_SCRATCH", room)
        w = rawphys.World(0, "fp64")
        w.load_batch(batch)
        w.sync()
        before = w.kernel_launches()
        results.append(w.adjoint(3, last, target, checkpoint_every=2, substeps=4))
        launches.append(w.kernel_launches() - before)
        w.close()
    # two segments of 8 and 4 substeps: two scalar passes (all frames; the first segment again), and per
    # group of substeps and turn a taping and a reverse sweep
    assert launches[0] == 2 + 2 * 2
    assert launches[1] == 2 + 2 * 6 * (8 + 4)
    assert launches[0] < launches[2] < launches[1]
    for res in results[1:]:
        for k in ("loss",) + KEYS:
            assert np.array_equal(res[k], results[0][k]), k
