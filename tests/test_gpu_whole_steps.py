"""GPU checks of whole steps taken in one launch (small handles with reused
lists): the same bits as the step's stages launched one by one.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

from test_gpu_lists import state, with_skin

pytestmark = pytest.mark.gpu


def moving(m, tension, obstacle):
    """The first m particles of a block in motion, some in free flight."""
    sc = scenes.dam_break(32, 32, 25, (0.0, 0.0, 0.0), (0.6, 0.6, 0.6), m, "whole", 1, obstacle=obstacle)
    rng = np.random.default_rng(m)
    p = P.SimulationParameters.from_buffer_copy(bytes(sc.params))
    p.numParticles = m
    p.tensionCoefficient = 0.0728 if tension else 0.0
    v = rng.uniform(-1.0, 1.0, (m, 3)).astype(np.float32)
    return scenes.Scene("whole", p, sc.options, sc.positions[:m].copy(), v, sc.boundary)


# a lone particle, the edges of a warp and of a block, a ragged grid, the
# most particles that take the form and one more (which does not)
@pytest.mark.parametrize("m, tension, obstacle", [
    (1, True, False), (31, False, False), (33, True, True), (127, True, False), (128, False, False),
    (129, True, False), (5000, True, True), (24575, False, False), (24576, True, False), (24577, True, False)])
def test_whole_steps_equal_separate_stages(sphlib, m, tension, obstacle):
    """40 steps by one call (more than one launch takes), by 40 calls, and
    with every stage a launch of its own (stage timing)."""
    sc = moving(m, tension, obstacle)
    outs = []
    for form in ("staged", "one call", "single"):
        with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, 0.1),
                                       sc.boundary) as sim:
            if form == "staged":
                sim.set_stage_timing(40)
            if form == "single":
                for _ in range(40):
                    sim.Advance()
            else:
                sim.step(count=40)
            assert sim.GetNumTimesSteps() == 40
            outs.append(state(sphlib, sim) | {"builds": sim.neighbour_builds(), "surface": sim.surface_particles()})
    for other in outs[1:]:
        for k in outs[0]:
            np.testing.assert_array_equal(other[k], outs[0][k], err_msg=k)
