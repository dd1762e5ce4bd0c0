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
