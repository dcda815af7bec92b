"""GPU boundary maps whose wall-viscosity terms lie next to a rounding
boundary: the term is the double product rounded once, as the reference's
host code forms it, also where two single-precision products could not tell
which way that goes.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P

pytestmark = pytest.mark.gpu

F = np.float32
NODES = 16


def desc(t):
    """A sphere on a lattice out of step with the nodes; in the t listed below
    a term next to a boundary changes a node's sum."""
    h = F(0.02) + F(0.0005) * F(t % 400)
    sp, ps = h * (F(0.23) + F(0.00137) * F(t % 31)), h * (F(0.41) + F(0.00311) * F(t % 37))
    start = (F(0.01), F(0.02), F(0.03))
    w = F(NODES - 1) * sp
    d = P.BoundaryDesc()
    for a in range(3):
        d.gridStart[a] = float(start[a])
        d.gridEnd[a] = float(start[a] + sp * F(NODES - 0.5))
    d.gridSpacing, d.restDistance, d.compactSupport, d.particleSpacing = float(sp), float(h), float(h), float(ps)
    d.particleMass = d.restDensity = d.viscosity = 1.0
    d.numShapes = 1
    d.shapes[0].kind = P.SHAPE_SPHERE
    values = (start[0] + F(0.5) * w, start[1] + F(0.45) * w, start[2] + F(0.5) * w, F(0.3) * w + F(0.0003) * F(t // 400))
    for k, v in enumerate(values):
        d.shapes[0].p[k] = float(v)
    return d


@pytest.mark.parametrize("t", [45271, 61615, 67783, 84509, 105015, 141675, 162772, 202258])
def test_viscosity_is_the_double_product_rounded_once(sphlib, orc, t):
    d = desc(t)
    assert d.dims() == (NODES,) * 3
    dist, dens, visc = sphlib.boundary_maps(d)
    bm = orc.boundary_maps(d)
    np.testing.assert_array_equal(dist, bm.dist)
    np.testing.assert_array_equal(visc, bm.visc)
