"""GPU checks of batched steps in which some scenes sort and others reuse
their lists: only the sorting scenes' particles go through the sort, and each
scene's state and tables are those of the scene run alone, step by step.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import scenes

from test_gpu_batch import check_scene
from test_gpu_lists import with_skin

pytestmark = pytest.mark.gpu


def read(sphlib, sim):
    h, ids, start, end = sim.cells()
    return dict(pos=sim.positions(), vel=sim.velocities(), rho=sim.read(sphlib.FIELD_DENSITY),
                acc=sim.read(sphlib.FIELD_ACCELERATION), hash=h, ids=ids, start=start, end=end)


def block(dims, speed, seed):
    sc = scenes.dam_break(*dims, (0.1, 0.1, 0.1), (0.6, 0.6, 0.6), seed, "block", 1)
    sc.velocities[:] = np.random.default_rng(seed).uniform(-speed, speed, sc.velocities.shape).astype(np.float32)
    return sc


# one scene; a scene at rest before, between and after moving ones; single particles
@pytest.mark.parametrize("shape", [
    [((9, 7, 5), 1.0)],
    [((9, 7, 5), 0.0), ((16, 16, 8), 3.0), ((5, 5, 5), 0.0), ((11, 3, 4), 15.0), ((8, 8, 8), 0.0)],
    [((1, 1, 1), 5.0), ((16, 8, 8), 0.0), ((1, 1, 1), 0.0), ((12, 12, 12), 2.0)]])
def test_scenes_that_sort_beside_scenes_that_reuse(sphlib, shape):
    scs = [block(d, v, 3 + k) for k, (d, v) in enumerate(shape)]
    alone = [sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, 0.1)) for sc in scs]
    try:
        with sphlib.ParticleSimulation.batch(scs, with_skin(scs[0], 0.1)) as sim:
            fp, fc = sim.scene_ranges()
            for step in range(12):
                sim.step()
                for a in alone:
                    a.step()
                if step % 3 == 2:  # (a read rebuilds stale tables: not after every step)
                    b = read(sphlib, sim)
                    for k, a in enumerate(alone):
                        check_scene(k, fp, fc, b, read(sphlib, a))
            assert sim.neighbour_builds() == sum(a.neighbour_builds() for a in alone)
    finally:
        for a in alone:
            a.close()
