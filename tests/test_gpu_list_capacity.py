"""GPU checks of the reused lists at large skins and in dense packings: a
list's capacity follows the candidates of the fluid at rest, and above a skin
of 0.25 the density stage records which candidates lie within h, a bit each,
32 to a word.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

from test_gpu_list_forms import cluster
from test_gpu_lists import state, with_skin
from test_gpu_step import check_step
from test_gpu_whole_steps import moving

pytestmark = pytest.mark.gpu


def denser(sc, factor):
    """The same positions with `factor` times as many particles in a volume at rest."""
    p = P.SimulationParameters.from_buffer_copy(bytes(sc.params))
    p.particleMass = float(np.float32(p.particleMass / factor))
    return scenes.Scene(sc.name, p, sc.options, sc.positions, sc.velocities)


# a word of eight groups and its edges; the capacities 184 (skin 0.4), 244
# (skin 0.1 at five times the density), 384 (the most) and one more of each
@pytest.mark.parametrize("skin, factor, sizes", [
    (0.3, 1, (1, 4, 31, 32, 33, 64, 65, 97)), (0.4, 1, (183, 184, 185, 260)), (0.25, 1, (33, 97, 132)),
    (0.1, 5, (96, 97, 200, 224, 225, 300)), (0.4, 9, (130, 384, 385, 500)), (0.05, 20, (384, 385))])
def test_reusing_steps_at_the_edges_of_a_capacity(sphlib, orc, skin, factor, sizes):
    for m in sizes:
        sc = denser(cluster(m, m), factor)
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, skin)) as sim:
            for k in range(3):
                x0, v0 = sim.positions(), sim.velocities()
                sim.Advance()
                check_step(orc, scenes.Scene("cluster", sc.params, sc.options, x0, v0), state(sphlib, sim), None)
            assert sim.neighbour_builds() == 1, m  # the second and third step walked the lists


@pytest.mark.parametrize("m, tension, obstacle", [(1, True, False), (129, True, False), (5000, True, True),
                                                  (24576, False, False), (24577, True, False)])
def test_whole_steps_equal_separate_stages_with_masks(sphlib, m, tension, obstacle):
    sc = moving(m, tension, obstacle)
    outs = []
    for staged in (True, False):
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, 0.4),
                                       sc.boundary) as sim:
            if staged:
                sim.set_stage_timing(40)
            sim.step(count=40)
            outs.append(state(sphlib, sim) | {"builds": sim.neighbour_builds(), "surface": sim.surface_particles()})
    for k in outs[0]:
        np.testing.assert_array_equal(outs[1][k], outs[0][k], err_msg=k)


@pytest.mark.parametrize("skin", [0.3, 0.4])
def test_a_batch_with_masks_equals_its_scenes_alone(sphlib, skin):
    many = [moving(m, False, ob) for m, ob in ((1000, False), (25000, True), (77, False))]
    o = with_skin(many[0], skin)
    with sphlib.ParticleSimulation.batch(many, o) as batch:
        batch.step(count=12)
        first, _ = batch.scene_ranges()
        x, v = batch.positions(), batch.velocities()
    for k, sc in enumerate(many):
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, o, sc.boundary) as sim:
            sim.step(count=12)
            np.testing.assert_array_equal(x[first[k]:first[k + 1]], sim.positions(), err_msg=str(k))
            np.testing.assert_array_equal(v[first[k]:first[k + 1]], sim.velocities(), err_msg=str(k))


def test_timing_the_force_after_a_building_step_reads_this_steps_masks(sphlib):
    """The masks of a step that built the lists are not written by it: the
    timed launches get theirs first, and the state is as the step left it."""
    sc = moving(25000, False, False)
    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, 0.4)) as sim:
        sim.step(count=1)
        before = state(sphlib, sim)
        assert sim.neighbour_builds() == 1
        assert sim.time_kernel("force", 3) > 0.0 and sim.time_kernel("density", 3) > 0.0
        after = state(sphlib, sim)
    for k in before:
        np.testing.assert_array_equal(after[k], before[k], err_msg=k)
