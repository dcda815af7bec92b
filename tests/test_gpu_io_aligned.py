"""GPU checks of reads into and writes from host memory at any byte.  Floats
off their 4-byte boundary go through a device buffer and a copy, also where
the memory is page-locked and a kernel could reach it.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import params as P
from cudasphnew_gb300 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def two_scale_tank():
    sc = scenes.dam_break(9, 8, 7, (0.0, 0.0, 0.0), (0.5, 0.5, 0.5), 5, "io", 1)
    o = P.Options.from_buffer_copy(bytes(sc.options))
    for a in range(3):
        o.splitMin[a], o.splitMax[a] = 0.02, 0.07
    return sc, o


# 16 bytes: vector stores; 4 and 12: single floats; 1, 2, 3: off the boundary
@pytest.mark.parametrize("off", [0, 4, 12, 16, 1, 2, 3])
@pytest.mark.parametrize("pinned", [True, False])
def test_reads_and_writes_at_any_byte(sphlib, off, pinned):
    sc, o = two_scale_tank()
    L = sphlib.load()
    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, o) as sim:
        sim.step(sphlib.SPH_STEP_TWO_SCALE, 2)
        for field in (sphlib.FIELD_VERTEX_DATA, sphlib.FIELD_VELOCITY, sphlib.FIELD_SUB_VERTEX_DATA):
            want = sim.read(field)
            raw = torch.zeros(want.nbytes + 64, dtype=torch.uint8, pin_memory=pinned)
            sphlib.check(L.sph_read(sim._h, field, raw.data_ptr() + off, want.nbytes))
            got = raw.numpy()
            np.testing.assert_array_equal(got[off:off + want.nbytes], want.view(np.uint8).ravel())
            assert not got[:off].any() and not got[off + want.nbytes:].any()
        rng = np.random.default_rng(off)
        for field in (sphlib.FIELD_VERTEX_DATA, sphlib.FIELD_VELOCITY):
            a = rng.uniform(0.1, 0.4, (sim.n, 3)).astype(np.float32)
            raw = torch.zeros(a.nbytes + 64, dtype=torch.uint8, pin_memory=pinned)
            raw.numpy()[off:off + a.nbytes] = a.view(np.uint8).ravel()
            sphlib.check(L.sph_write(sim._h, field, raw.data_ptr() + off, a.nbytes))
            sim.synchronize()
            np.testing.assert_array_equal(sim.read(field), a)
