"""GPU check of steps on a stream that the caller is capturing: one step is
recorded, many steps in one call are refused at every size of handle.
"""
import numpy as np
import pytest

from cudasphnew_gb300 import scenes

from test_gpu_lists import with_skin

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_many_steps_are_refused_under_capture(sphlib):
    sc = scenes.dam_break(16, 16, 16, (0.0, 0.0, 0.0), (0.5, 0.5, 0.5), 3, "capture", 1)
    with sphlib.ParticleSimulation(sc.params, sc.positions, sc.velocities, with_skin(sc, 0.1)) as sim:
        st = torch.cuda.Stream()
        sim.set_stream(st.cuda_stream)
        sim.step(count=2)
        sim.synchronize()
        x0, steps = sim.positions(), sim.GetNumTimesSteps()
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st):
            with pytest.raises(sphlib.SphError) as e:
                sim.step(count=3)
        assert e.value.status == 2  # SPH_ERR_CUDA
        assert sim.GetNumTimesSteps() == steps
        np.testing.assert_array_equal(sim.positions(), x0)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            sim.step(count=1)
        g.replay()
        torch.cuda.synchronize()
        once = sim.positions()
    assert np.abs(once - x0).max() > 0
