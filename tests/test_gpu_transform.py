"""The FP64 hull transform's threads per collider follow the hulls' size: worlds of one kind of hull (8, 20, 64 and 80
vertices or faces) and of small ones beside spheres equal the oracle bit for bit."""
import numpy as np
import pytest

import rawphys
from oracle.oracle import Oracle
from rawphys import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["cube", "icosahedron", "cylinder32", "icosphere42", "spheres"])
def test_worlds_of_one_kind_of_hull(mesh):
    rng = np.random.default_rng(5)
    b = S._Builder("kind-" + mesh)
    for i in range(9):
        q = rng.normal(size=4)
        kw = dict(rot=tuple(q / np.linalg.norm(q)), mass=1.0, fixed=i == 0)
        p = (0.3 * (i % 3), 0.9 * i, 0.2 * (i % 2))
        if mesh == "spheres" and i % 2:
            b.body([S.Collider("sphere", radius=0.5)], p, **kw)
        else:
            b.hull_body("cube" if mesh == "spheres" else mesh, (0.55, 0.5, 0.6), p, **kw)
    sc = b.finish(dt=1.0 / 60.0, substeps=10, pos_iters=1, collisions=True, steps=1)
    w = rawphys.World(0, "fp64")
    w.load(sc)
    w.step(8)
    o = Oracle("port").load(sc)
    o.step(8)
    assert np.array_equal(w.get_state(), o.get_state())
    w.close()
