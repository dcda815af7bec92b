"""GPU checks of the reused lists at large skins and in dense packings: a
list holds 480 candidates where there is room, rows of up to 64 places are
masked in a building step, and above a skin of 0.25 the density stage of a
reusing one records which candidates lie within h, a bit each, 32 to a word.
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


# a word of eight groups and its edges; rows of 32, 33, 64 and 65 places and
# more; the most candidates a list holds (480) and one more
@pytest.mark.parametrize("skin", [0.05, 0.1, 0.3, 0.4])
@pytest.mark.parametrize("sizes", [(1, 4, 31, 32, 33), (64, 65, 96, 97), (130, 255, 256, 257), (479, 480, 481, 600)])
def test_reusing_steps_at_the_edges_of_a_capacity(sphlib, orc, skin, sizes):
    for m in sizes:
        sc = cluster(m, m)
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, skin)) as sim:
            for k in range(3):
                x0, v0 = sim.positions(), sim.velocities()
                sim.Advance()
                check_step(orc, scenes.Scene("cluster", sc.params, sc.options, x0, v0), state(sphlib, sim), None)
            builds = sim.neighbour_builds()
        # a dense cluster flies apart: its second step may outrun the first one's lists
        assert builds >= 1 and (builds == 1 or m > 96), m


def row_of_particles(m, seed):
    """m particles within a support radius in x, in one row of cells (as many
    places in it), and a particle above them that has all of them in reach."""
    sc = scenes.dam_break(4, 4, 4, (0.0, 0.0, 0.0), (0.5, 0.5, 0.5), seed, "row", 1)
    h = float(sc.params.compactSupport)
    rng = np.random.default_rng(seed)
    x = np.full((m, 3), 0.2)
    x[:, 0] += np.linspace(-0.45, 0.45, m) * h + rng.uniform(-0.1, 0.1, m) * h / m
    x[:, 1:] += 0.05 * h * rng.uniform(-1.0, 1.0, (m, 2))
    x = np.concatenate([x, [[0.2, 0.2 + 0.3 * h, 0.2]]]).astype(np.float32)
    p = P.SimulationParameters.from_buffer_copy(bytes(sc.params))
    p.numParticles = len(x)
    return scenes.Scene("row", p, sc.options, x, np.zeros_like(x))


@pytest.mark.parametrize("m", [30, 31, 32, 33, 34, 62, 63, 64, 65, 66, 100])
@pytest.mark.parametrize("skin", [0.05, 0.4])
def test_building_steps_over_long_rows_equal_the_per_step_search(sphlib, m, skin):
    """Rows of up to 32, 64 and more places: one mask word, two, none."""
    sc = row_of_particles(m, m)
    outs = []
    for s in (0.0, skin):
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, s)) as sim:
            sim.Advance()
            outs.append(state(sphlib, sim))
    for k in outs[0]:
        np.testing.assert_array_equal(outs[1][k], outs[0][k], err_msg=k)


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
