"""GPU checks of the reused lists' storage: groups of four candidates with a
partly filled last one, more candidates than a list holds (the rows' windows
instead), and steps that search without building because each one moves some
particle past the rebuild distance.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

from test_gpu_lists import moving_scene, state, with_skin
from test_gpu_step import check_step

pytestmark = pytest.mark.gpu


def cluster(m, seed):
    """m particles within half a support radius of one another (each is every
    other's neighbour, and m candidates are on every list) and a loose one."""
    sc = scenes.dam_break(4, 4, 4, (0.0, 0.0, 0.0), (0.5, 0.5, 0.5), seed, "cluster", 1)
    rng = np.random.default_rng(seed)
    h = float(sc.params.compactSupport)
    x = rng.normal(size=(m, 3))
    x *= 0.25 * h * rng.uniform(0.2, 1.0, (m, 1)) / np.linalg.norm(x, axis=1, keepdims=True)
    x = np.concatenate([x + 0.21, [[0.4, 0.4, 0.4]]]).astype(np.float32)
    p = P.SimulationParameters.from_buffer_copy(bytes(sc.params))
    p.numParticles = len(x)
    return scenes.Scene("cluster", p, sc.options, x, np.zeros_like(x))


# one group and its edges, 16 groups, the most a list holds (96) and one more
@pytest.mark.parametrize("m", [1, 3, 4, 5, 63, 64, 65, 95, 96, 97, 200])
def test_reusing_step_at_the_edges_of_a_list(sphlib, orc, m):
    sc = cluster(m, m)
    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, sc.options) as sim:
        for k in range(3):
            x0, v0 = sim.positions(), sim.velocities()
            sim.Advance()
            check_step(orc, scenes.Scene("cluster", sc.params, sc.options, x0, v0), state(sphlib, sim), None)
        assert sim.neighbour_builds() == 1  # the second and third step walked the lists


def test_fast_steps_search_and_build_no_lists(sphlib):
    """Every step moves particles past the rebuild distance: after the first
    build the steps search, bit for bit as a handle without lists; once the
    motion stops, the lists are built again and reused."""
    sc = moving_scene(15.0)
    outs = []
    for skin in (0.0, 0.1):
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, skin)) as sim:
            sim.step(count=6)
            outs.append(state(sphlib, sim))
            if skin > 0:
                assert sim.neighbour_builds() == 1
                np.testing.assert_array_equal(sim.surface_particles(), flags)
                sim.write(sphlib.FIELD_VELOCITY, np.zeros_like(sc.positions))
                sim.step(count=4)
                assert sim.neighbour_builds() == 2
            else:
                flags = sim.surface_particles()
    for k in outs[0]:
        np.testing.assert_array_equal(outs[1][k], outs[0][k], err_msg=k)
