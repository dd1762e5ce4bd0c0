"""The scene-resident solve kernel at the edges of its ranges: its two size classes (up to and beyond 128
bodies), chunks of 32 nodes, scenes with more levels than it counts, several position iterations."""
import numpy as np
import pytest

import rawphys
from oracle.oracle import Oracle
from rawphys import scenes

pytestmark = pytest.mark.gpu


def _scenes():
    # a stack of n cubes and its floor: n + 1 bodies (126..128 cross the size classes); a chain of 260 links
    # is deeper than the kernel's 256 levels
    out = [scenes.stack_scene(n, seed=n) for n in (1, 2, 31, 32, 33, 126, 127, 128, 300)]
    out += [scenes.chain_scene(n, joint, seed=n) for n, joint in ((8, "hinge"), (33, "spherical"), (64, "hinge"), (260, "spherical"))]
    return out + [scenes.spring_scene(seed=1)]


def _world(precision, scs, iters, frames=2):
    w = rawphys.World(0, precision)
    first = [w.load(sc, 0 if k == 0 else w.new_scene()) for k, sc in enumerate(scs)]
    w.simulate(1.0 / 60.0, 20, iters, True, frames)
    state = w.get_state()
    w.close()
    return [state[f:f + sc.num_bodies] for f, sc in zip(first, scs)]


@pytest.mark.parametrize("iters", [1, 2])
def test_exact_solves_equal_the_oracle(iters):
    scs = _scenes()
    for sc, got in zip(scs, _world("fp64", scs, iters)):
        o = Oracle("port").load(sc)
        o.step(2, pos_iters=iters, collisions=True)
        assert np.array_equal(got, o.get_state()), (sc.name, sc.num_bodies)


@pytest.mark.parametrize("iters", [1, 2])
def test_fp32_solves_equal_the_sweep_kernels(iters):
    # a scene of more than 640 bodies puts a world on the sweep kernels, which keep the state in global
    # memory: the same operations with the same roundings, so the same bits
    scs = _scenes()
    big = scenes.stack_scene(640, seed=5)
    for sc, a, b in zip(scs, _world("fp32", scs, iters), _world("fp32", scs + [big], iters)):
        assert np.array_equal(a, b), (sc.name, sc.num_bodies)
