"""How a batch's sweeps spread scenes over warps and CTAs by default: the same results as a warp for every scene, on
both sides of the size from which a scene gets a CTA."""
import numpy as np
import pytest

import rawphys
from rawphys import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("order", ["coloured", "reference"])
def test_wide_scenes_on_a_cta_equal_warps(precision, order):
    # stacks of 93 to 96 cubes and their floor (94 to 97 bodies), a pile, chains below and above cost 96, and
    # in the reference order a scene of more than 640 bodies, which puts the world on the sweep kernels
    scs = [S.stack_scene(n, seed=n) for n in (2, 93, 94, 95, 96)] + [S.random_pile_scene(140, seed=7)]
    scs += [S.chain_scene(n, joint, seed=n) for n, joint in ((9, "hinge"), (12, "spherical"), (40, "hinge"))]
    if order == "reference":
        scs.append(S.stack_scene(650, seed=5))
    states = []
    for assignment in (0, 1000000):
        w = rawphys.World(0, precision)
        w.set_sweep_order(order)
        w.set_sweep_assignment(assignment)
        for k, sc in enumerate(scs):
            w.load(sc, 0 if k == 0 else w.new_scene())
        w.simulate(1.0 / 60.0, 10, 2, True, 2)
        states.append(w.get_state())
        w.close()
    assert np.array_equal(*states)


@pytest.mark.parametrize("solved", [True, False])
def test_autotune_times_sweep_layouts_only_where_sweeps_run(solved):
    # phased, persistent and three other transform groups; five more sweep assignments in the coloured order
    w = rawphys.World(0, "fp32")
    for k in range(4):
        w.load(S.stack_scene(4, seed=k), 0 if k == 0 else w.new_scene())
    if not solved:
        w.set_sweep_order("coloured")
    w.step(1)
    before = w.kernel_launches()
    w.step(10)
    frame = (w.kernel_launches() - before) // 10
    before = w.kernel_launches()
    choice = w.autotune(frames=4)
    frames = (w.kernel_launches() - before) / frame
    trials = 2 * (1 + 4)   # each candidate twice, a warm-up and four frames (and the state's upload)
    if choice["mode"] == "phased":
        assert (4 if solved else 9) * trials <= frames <= (4 if solved else 9) * trials + 3 * trials
    if solved:
        assert choice["batch_sweep_assignment"] == "CTA for wide scenes"
    w.close()
