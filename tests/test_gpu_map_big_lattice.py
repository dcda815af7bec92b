"""GPU boundary maps over a ghost lattice too large for its bits to be kept
(2^26 words): each node then tests the lattice points around it itself.  The
oracle would walk the whole lattice, so the nodes next to the solid are
restated here, term by term.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P

pytestmark = pytest.mark.gpu

F = np.float32
PS, HS = F(1 / 64), F(2.3 / 64)  # lattice pitch, support


def desc(pitches):
    """3^3 nodes, `pitches` lattice pitches apart, and a sphere around node 0 that ends next to its neighbours."""
    d = P.BoundaryDesc()
    sp = F(pitches) * PS
    for a in range(3):
        d.gridStart[a] = float(F(0.37) * F(a + 1))
        d.gridEnd[a] = float(F(d.gridStart[a]) + F(2.5) * sp)
    d.gridSpacing, d.restDistance, d.compactSupport, d.particleSpacing = float(sp), float(HS), float(HS), float(PS)
    d.particleMass = d.restDensity = d.viscosity = 1.0
    d.numShapes = 1
    d.shapes[0].kind = P.SHAPE_SPHERE
    for k, v in enumerate((*[d.gridStart[a] for a in range(3)], float(sp + F(0.3) * HS))):
        d.shapes[0].p[k] = v
    return d


def node_sums(d, node):
    h, ps = F(d.compactSupport), F(d.particleSpacing)
    hd = float(h)
    rho_coeff, vis_coeff = 64.0 * 3.14159265358979323846, 3.14159265358979323846
    for _ in range(9):
        rho_coeff *= hd
    for _ in range(6):
        vis_coeff *= hd
    rho_coeff, vis_coeff = F(315.0 / rho_coeff), 45.0 / vis_coeff
    margin = h + ps
    lat = [F(d.gridStart[a]) - margin for a in range(3)]
    x = [F(d.gridStart[a]) + F(d.gridSpacing) * F(node[a]) for a in range(3)]
    c = [float(d.shapes[0].p[k]) for k in range(4)]
    lo = [int(np.floor((x[a] - h - lat[a]) / ps)) - 1 for a in range(3)]
    hi = [int(np.floor((x[a] + h - lat[a]) / ps)) + 1 for a in range(3)]
    rho = vis = F(0)
    for k in range(max(lo[2], 0), hi[2] + 1):
        for j in range(max(lo[1], 0), hi[1] + 1):
            for i in range(max(lo[0], 0), hi[0] + 1):
                g = [lat[a] + F(n) * ps for a, n in enumerate((i, j, k))]
                dx, dy, dz = (float(g[a]) - c[a] for a in range(3))
                if F(np.sqrt(dx * dx + dy * dy + dz * dz) - c[3]) > 0:
                    continue
                ex, ey, ez = (g[a] - x[a] for a in range(3))
                sq = ex * ex + ey * ey + ez * ez
                diff = h * h - sq
                if diff >= 0:
                    rho = rho + rho_coeff * diff * diff * diff
                dist = np.sqrt(sq)
                if dist <= h:
                    vis = vis + F(vis_coeff * float(h - dist))
    return rho, vis


@pytest.mark.parametrize("pitches", [600, 650])  # 38 * 1207^2 words: bits; 41 * 1307^2: none
def test_maps_with_and_without_the_lattice_bits(sphlib, pitches):
    d = desc(pitches)
    assert d.dims() == (3, 3, 3)
    dist, dens, visc = sphlib.boundary_maps(d)
    near = {(1, 0, 0), (0, 1, 0), (0, 0, 1)}
    for k in range(3):
        for j in range(3):
            for i in range(3):
                want = node_sums(d, (i, j, k)) if (i, j, k) in near else (F(0), F(0))
                assert (dens[k, j, i], visc[k, j, i]) == want, (i, j, k)
                assert ((i, j, k) in near) == (want[0] > 0) == (dist[k, j, i] > -HS)
