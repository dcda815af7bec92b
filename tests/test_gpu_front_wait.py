"""GPU checks of a sort whose device-side waits give up part of the way: the
wait limit (polls of a block at a grid barrier) is shortened on the host, so
blocks start, wait and leave in many orders.
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
    """(on a handle that has stepped before)"""
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


FORMS = {
    "search": dict(dims=(32, 32, 32), skin=0.0),
    "lists": dict(dims=(32, 32, 32), skin=0.1),
    "whole steps": dict(dims=(16, 16, 16), skin=0.1),
    "timed stages": dict(dims=(32, 32, 32), skin=0.1, timed=1),
    "cell-relative": dict(dims=(16, 16, 16), skin=0.0, relative=1),
    "staged force": dict(dims=(16, 16, 16), skin=0.0, variant=3),
    "batch, search": dict(dims=(16, 16, 16), skin=0.0, scenes=3),
    "batch, lists": dict(dims=(16, 16, 16), skin=0.1, scenes=3),
    "two-scale": dict(dims=(16, 16, 16), skin=0.0, mode=1),
    "learned, search": dict(dims=(16, 16, 16), skin=0.0, mode=3),
    "learned, lists": dict(dims=(16, 16, 16), skin=0.1, mode=3),
}


@pytest.mark.parametrize("before", [0, 3])
@pytest.mark.parametrize("form", list(FORMS))
def test_a_step_whose_sort_gave_up_changes_nothing(sphlib, form, before):
    """Every wait gives up at its first poll, on the handle's first step and
    after some good ones: the condition is reported once, the state stays as
    it was, and steps from there on are good ones."""
    f = FORMS[form]
    mode = f.get("mode", sphlib.SPH_STEP_PLAIN)
    sc, o = tank(*f["dims"], f["skin"])
    o.cellRelative = f.get("relative", 0)
    if mode == sphlib.SPH_STEP_TWO_SCALE:
        for a in range(3):
            o.splitMin[a], o.splitMax[a] = 0.05, 0.2

    def handle():
        if "scenes" in f:
            sim = sphlib.ParticleSimulation.batch([tank(8 + 2 * k, 16, 16, f["skin"], k + 1)[0]
                                                   for k in range(f["scenes"])], o)
        else:
            sim = sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, o)
        if mode == sphlib.SPH_STEP_LEARNED:
            sim.load_corrector(np.zeros(sphlib.CORRECTOR_FLOATS, np.float32))
        if "variant" in f:
            sim.set_tuning(forceVariant=f["variant"])
        if "timed" in f:
            sim.set_stage_timing(4)
        for _ in range(before):
            sim.step(mode, 1)
        if before and f["skin"] > 0:  # so far that the next step does not reuse its lists: it sorts, and waits
            sim.write_state(sim.positions() + np.float32(1e-3), sim.velocities())
        sim.synchronize()
        return sim

    def particles(sim, stepped):
        out = [sim.positions(), sim.velocities()]
        return out + [sim.read(k) for k in (sphlib.FIELD_DENSITY, sphlib.FIELD_ACCELERATION) if stepped]

    with handle() as sim, handle() as ref:
        was = particles(sim, before)
        os.environ["SPH_SCAN_WAIT_LIMIT"] = "-1"
        try:
            for _ in range(2):  # the second sorts nothing: the first's give-up is not reported yet
                sim.step(mode, 1)
            with pytest.raises(sphlib.SphError) as e:
                sim.synchronize()
            assert e.value.status == WAIT
        finally:
            del os.environ["SPH_SCAN_WAIT_LIMIT"]
        sim.synchronize()  # reported once
        for got, want in zip(particles(sim, before), was):
            np.testing.assert_array_equal(got, want)
        if f["skin"] > 0:  # the step that follows builds the lists
            for s in (sim, ref):
                s.write_state(was[0] + np.float32(1e-3), was[1])
        for s in (sim, ref):
            s.step(mode, 1)
        for got, want in zip(particles(sim, True), particles(ref, True)):
            np.testing.assert_array_equal(got, want)
            assert np.isfinite(got).all()
