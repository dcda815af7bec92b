"""GPU boundary maps of scenes whose lengths are so small or so large that
their squares leave single precision's range: the distances are the double
ones rounded once, as at any other scale.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P

pytestmark = pytest.mark.gpu


def desc(unit, kind):
    nodes, h = 20, 0.25
    w = (nodes - 1) * h / 4
    p = {P.SHAPE_SPHERE: (0.5 * w, 0.45 * w, 0.5 * w, 0.3 * w),
         P.SHAPE_CONE: (0.5 * w, 0.5 * w, 0.2 * w, 0.25 * w, 0.5 * w)}[kind]
    d = P.BoundaryDesc()
    for a in range(3):
        d.gridStart[a] = unit * 0.01 * (a + 1)
        d.gridEnd[a] = d.gridStart[a] + unit * (w + h / 8)
    d.gridSpacing, d.restDistance, d.compactSupport, d.particleSpacing = unit * h / 4, unit * h, unit * h, unit * h / 2
    d.particleMass = d.restDensity = d.viscosity = 1.0
    d.numShapes = 1
    d.shapes[0].kind = kind
    for k, v in enumerate(p):
        d.shapes[0].p[k] = unit * v
    return d


@pytest.mark.parametrize("kind", [P.SHAPE_SPHERE, P.SHAPE_CONE])
@pytest.mark.parametrize("unit", [1e-24, 1e-21, 1e-18, 1e-14, 1e-6, 1.0, 1e6, 1e14, 1e18, 1e20, 1e24])
def test_distances_at_any_scale(sphlib, orc, unit, kind):
    d = desc(unit, kind)
    np.testing.assert_array_equal(sphlib.boundary_maps(d)[0], orc.boundary_maps(d).dist)
