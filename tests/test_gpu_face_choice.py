"""The reference face of nearly parallel faces: the warp kernels decide it in FP32 from |m - n|^2 beyond a margin and in
FP64 within it, the persistent form's general code always in FP64. Both take the same face, at tilts on either
side of the margin (about 1e-5 rad)."""
import numpy as np
import pytest

import rawphys
from rawphys import scenes as S

pytestmark = pytest.mark.gpu


def _tilted(mesh, seed, count):
    # pairs in one scene each: a fixed hull with a face up, a body 1 mm into it, tilted by 1e-8 to 1e-2 rad, both
    # turned about y, and every third pair turned as a whole (the face normals then have roundings of their own)
    rng = np.random.default_rng(seed)
    out = []
    for k in range(count):
        b = S._Builder("tilt%d" % k)
        a, t = rng.uniform(0.0, 2.0 * np.pi, size=2)
        tilt = 10.0 ** rng.uniform(-8.0, -2.0)
        axis = np.array([np.cos(t), 0.0, np.sin(t)])
        turn = np.array([0.0, np.sin(a / 2), 0.0, np.cos(a / 2)])
        lean = np.append(axis * np.sin(tilt / 2), np.cos(tilt / 2))
        whole = rng.normal(size=4) if k % 3 == 0 else np.array([0.0, 0.0, 0.0, 1.0])
        whole /= np.linalg.norm(whole)
        height = 0.5 + 0.5 * rng.uniform(0.8, 1.2)
        scale = 2.0 * (height - 0.5)
        p = np.array([rng.uniform(-0.2, 0.2), height - 0.001, rng.uniform(-0.2, 0.2)])
        b.hull_body("cube", (0.5, 0.5, 0.5), (0.0, 0.0, 0.0), rot=tuple(whole), fixed=True)
        b.hull_body(mesh, (0.5 * scale,) * 3, tuple(_rotate(whole, p)), rot=tuple(_mul(whole, _mul(lean, turn))), mass=1.0)
        out.append(b.finish(dt=1.0 / 60.0, substeps=1, pos_iters=1, collisions=True, steps=1))
    return out


def _mul(a, b):
    x, y, z, w = a
    return np.array([w * b[0] + x * b[3] + y * b[2] - z * b[1], w * b[1] - x * b[2] + y * b[3] + z * b[0],
                     w * b[2] + x * b[1] - y * b[0] + z * b[3], w * b[3] - x * b[0] - y * b[1] - z * b[2]])


def _rotate(q, v):
    return _mul(_mul(q, np.append(v, 0.0)), np.array([-q[0], -q[1], -q[2], q[3]]))[:3]


@pytest.mark.parametrize("mesh", ["cube", "cylinder32"])
def test_nearly_parallel_faces_choose_as_fp64_does(mesh):
    scs = _tilted(mesh, 3, 500)
    found = []
    for mode in ("phased", "persistent"):
        w = rawphys.World(0, "fp32")
        w.set_mode(mode)
        first = [w.load(sc, 0 if k == 0 else w.new_scene()) for k, sc in enumerate(scs)]
        # a substep of 1 us: the poses the contacts are found at are the given ones to rounding
        w.simulate(1e-6, 1, 1, True, 1)
        found.append([w.last_contacts(k)[1] for k in range(len(scs))])
        w.close()
    touching = 0
    for k, (a, b) in enumerate(zip(*found)):
        assert a.shape == b.shape, k
        touching += len(a) > 0
        # anchors and normal: the other face as reference would give other points (the body's corners instead of
        # their projections, in another order); FP32 rounding of metre-sized values is 6e-8
        assert len(a) == 0 or np.abs(a[:, :9] - b[:, :9]).max() <= 1e-6, k
    assert touching > 400
