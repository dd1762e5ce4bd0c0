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
