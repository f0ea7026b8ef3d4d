"""The mass the FP32 paths miss has no direction: over many steps of a steady flow the
mean drift of many tracers stays within the resolution of the mass itself."""
import numpy as np
import pytest

from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP32_COMP])
def test_no_steady_drift(precision):
    """1000 steps, 24 tracers over thick layers with thin ones on top: a mass is an
    FP64 number (2.2e-16 of itself), the mean of 24 is held to that; sums whose
    rounding leans one way drifted by 7e-16."""
    case = synth.make("stiff2048", nx=512, ny=256)
    t = gpu.TracerStep(case, precision=precision)
    t.start()
    t.sync()
    m0 = np.array(t.mass())
    t.run(1000)
    t.sync()
    drift = (np.array(t.mass()) - m0) / m0
    t.close()
    assert abs(drift.mean()) <= 2.2e-16
    assert np.abs(drift).max() <= 1e-15
