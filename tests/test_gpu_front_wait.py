"""GPU checks of a sort whose device-side waits give up part of the way: the
wait limit (polls of a block at a grid barrier) is shortened on the host, so
blocks start, wait and leave in many orders.  Each handle has stepped before.
"""
import os

import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

from test_gpu_lists import state, with_skin

pytestmark = pytest.mark.gpu

WAIT = 5  # SPH_ERR_DEVICE_WAIT


def tank(nx, ny, nz, skin, seed=1):
    sc = scenes.dam_break(nx, ny, nz, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), seed, "wait", 1)
    return sc, with_skin(sc, skin)


# more blocks than one in each form: whole steps, k_front with lists (above the
# whole steps' size), k_front alone, and the fine level's sort
@pytest.mark.parametrize("form, dims, skin", [("plain", (24, 24, 24), 0.1), ("plain", (32, 32, 32), 0.1),
                                              ("plain", (32, 32, 32), 0.0), ("two_scale", (24, 24, 24), 0.0)])
def test_waits_that_give_up_on_the_way_are_reported_and_recovered(sphlib, form, dims, skin):
    sc, o = tank(*dims, skin)
    if form == "two_scale":
        for a in range(3):
            o.splitMin[a], o.splitMax[a] = 0.05, 0.2
    mode = sphlib.SPH_STEP_TWO_SCALE if form == "two_scale" else sphlib.SPH_STEP_PLAIN

    def outcome(sim):
        sim.write_state(sc.positions, sc.velocities)
        sim.step(mode, 1)
        out = state(sphlib, sim)
        if form == "two_scale":
            out["children"] = sim.read(sphlib.FIELD_SUB_IDS)
            out["child positions"] = sim.read(sphlib.FIELD_SUB_VERTEX_DATA)[out["children"]]
        return out

    # far enough that lists are not reused from one state to the other
    shifted = sc.positions + np.float32(1e-3)

    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, o) as sim:
        sim.write_state(shifted, sc.velocities)
        sim.step(mode, 1)
        want = outcome(sim)
        given_up = 0
        for limit in (-1, 0, 1, 2, 4, 8, 16, 32, 64) * 4:
            sim.write_state(shifted, sc.velocities)
            os.environ["SPH_SCAN_WAIT_LIMIT"] = str(limit)
            try:
                sim.step(mode, 1)
                try:
                    sim.synchronize()
                except sphlib.SphError as e:
                    # (a particle may end outside the grid: the step's results are unspecified)
                    given_up += e.status == WAIT
            finally:
                del os.environ["SPH_SCAN_WAIT_LIMIT"]
            sim.synchronize()  # reported once
            got = outcome(sim)
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg="%s after limit %d" % (k, limit))
        assert given_up >= 4  # limit -1 always does
