"""GPU checks of the cell scan where cells far outnumber particles and where
its stretches end: grids of a few cells, of one stretch a warp or a block
more or less, and of millions, with particles in the first and last cells.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

pytestmark = pytest.mark.gpu


def scattered(side, n, skin):
    """n particles anywhere in a box of `side` (a few cells a side up), some in its first and last corner."""
    rng = np.random.default_rng(n)
    p = P.dam_break_params((0, 0, 0), (side,) * 3, n)
    x = rng.uniform(0.0, side, (n, 3))
    x[:4], x[4:8] = rng.uniform(0.0, 0.01, (4, 3)), side - rng.uniform(0.0, 0.01, (4, 3))
    o = P.default_options(gravity_axis=2, box_collision=True)
    o.neighbourSkin = skin
    return scenes.Scene("sparse", p, o, x.astype(np.float32), np.zeros((n, 3), np.float32))


def check_cells(sphlib, sc):
    g = sc.params
    dim = [int(d) for d in g.gridDim]
    with sphlib.ParticleSimulation(g, sc.positions, None, sc.options) as sim:
        for _ in range(2):  # the second finds the counts that the first has cleared
            sim.write_state(sc.positions, sc.velocities)
            sim.step(count=1)
            h, ids, start, end = sim.cells()
            # the hash as the kernels form it: rounded operations, truncation
            c = ((sc.positions - np.array(list(g.gridOrigin), np.float32)) / np.float32(g.gridSpacing)).astype(np.int64)
            want = c[:, 0] + dim[0] * (c[:, 1] + dim[1] * c[:, 2])
            order = np.argsort(want, kind="stable")
            np.testing.assert_array_equal(ids, order)
            np.testing.assert_array_equal(h, want[order])
            cells, first, count = np.unique(want[order], return_index=True, return_counts=True)
            np.testing.assert_array_equal(start[cells], first)
            np.testing.assert_array_equal(end[cells], first + count)
            empty = np.ones(len(start), bool)
            empty[cells] = False
            assert (start[empty] == start[empty][0]).all() and (end[empty] == end[empty][0]).all()


# cells a side: 8 .. 244 (14.5 million cells)
@pytest.mark.parametrize("side", [0.1, 0.15, 0.2, 0.5, 1.0, 1.6, 3.0, 6.0])
@pytest.mark.parametrize("n, skin", [(700, 0.0), (700, 0.1), (30000, 0.0), (30000, 0.1)])
def test_cell_tables_of_sparse_grids(sphlib, side, n, skin):
    check_cells(sphlib, scattered(side, n, skin))


# one, two and three passes of a block an SM (152) of 512 particles, and one particle more
@pytest.mark.parametrize("n", [77824, 77825, 155648, 155649, 233472, 233473])
def test_cell_tables_where_the_grid_takes_another_pass(sphlib, n):
    check_cells(sphlib, scattered(1.0, n, 0.0))
