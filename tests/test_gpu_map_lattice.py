"""GPU boundary maps against the oracle where the ghost lattice's rows end at
the edges of a 32-bit word, for each kind of solid and for several together.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P

pytestmark = pytest.mark.gpu

SPHERE, CONE, BOX = P.SHAPE_SPHERE, P.SHAPE_CONE, P.SHAPE_BOX


def desc(nodes, shapes):
    p = P.dam_break_params((0, 0, 0), (1, 1, 1), 4096)
    return P.obstacle_boundary(p, (0.013, -0.021, 0.005), nodes, shapes)


# rows of 2 * nodes / 4 + 7 lattice points: 31, 32, 33, then 64 and 65
@pytest.mark.parametrize("nodes", [48, 50, 52, 114, 116])
@pytest.mark.parametrize("kind", ["sphere", "cone", "box", "sphere+cone", "box+sphere"])
def test_maps_match_the_oracle(sphlib, orc, nodes, kind):
    w = (nodes - 1) * P.H / 4
    shapes = {SPHERE: (SPHERE, (0.013 + 0.5 * w, -0.021 + 0.45 * w, 0.005 + 0.5 * w, 0.3 * w)),
              CONE: (CONE, (0.013 + 0.6 * w, -0.021 + 0.5 * w, 0.005 + 0.2 * w, 0.25 * w, 0.5 * w)),
              BOX: (BOX, (0.013 + 0.5 * w, -0.021 + 0.5 * w, 0.005 + 0.5 * w, 0.4 * w, 0.35 * w, 0.41 * w))}
    names = {"sphere": SPHERE, "cone": CONE, "box": BOX}
    d = desc(nodes, [shapes[names[k]] for k in kind.split("+")])
    dist, dens, visc = sphlib.boundary_maps(d)
    bm = orc.boundary_maps(d)
    # the distance is the FP64 one rounded once, whatever decided that it was needed
    np.testing.assert_array_equal(dist, bm.dist)
    for got, ref in ((dens, bm.dens), (visc, bm.visc)):
        assert (np.abs(got - ref) <= 1e-6 * np.abs(ref)).all()
        assert np.abs(ref).max() > 0
