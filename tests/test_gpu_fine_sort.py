"""GPU checks of the fine level's counting sort at the edges of its grid: no
child at all, one parent's eight, a ragged number, and more children than the
launch has threads (each strides over several).
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, split", [((4, 4, 4), 0), ((1, 1, 1), 1), ((5, 7, 11), 385), ((32, 32, 16), 16384)])
def test_children_sorted_by_cell_in_list_order(sphlib, dims, split):
    sc = scenes.dam_break(*dims, (0.1, 0.1, 0.1), (0.6, 0.6, 0.6), 7, "fine", 1)
    o = P.Options.from_buffer_copy(bytes(sc.options))
    for a in range(3):  # the whole block splits, or nothing does
        o.splitMin[a], o.splitMax[a] = (-1.0, 2.0) if split else (5.0, 6.0)
    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, o) as sim:
        for step in range(2):
            sim.step(mode=sphlib.SPH_STEP_TWO_SCALE)
            c = sim.counts()
            assert c.numParticlesSplit == split and c.numSubParticles == 8 * split
            h, ids, start, end = sim.cells(1)
            listed = sim.read(sphlib.FIELD_SUB_IDS)
            np.testing.assert_array_equal(listed, np.arange(8 * split))
            # stable: (cell, place in the child list) ascends strictly
            key = h.astype(np.int64) * (8 * split + 1) + ids
            assert (np.diff(key) > 0).all()
            np.testing.assert_array_equal(np.sort(ids), listed)
            count = np.bincount(h, minlength=len(start))
            first = np.cumsum(count) - count
            np.testing.assert_array_equal(start, np.where(count > 0, first, -1))
            np.testing.assert_array_equal(end, np.where(count > 0, first + count, -1))
