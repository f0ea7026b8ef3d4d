"""What a step costs in windows away from the usual shapes: few layers, columns much
shallower than the layers the window has, few tracers.  Each bound lies between
what the launch that fits such a window takes and what one made for the usual
shapes took (ratios of times of one run, or of two windows of the same work).
"""
import numpy as np
import pytest

from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


def window(nx, ny, nz, ntr, **kw):
    d = dict(seed=91, ntr=ntr, depth=(3.0, 5.0 * nz - 1.0), land_frac=0.15, cell=(400.0, 900.0),
             curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1), tracers=("logn", 1e-2, 10.0))
    d.update(kw)
    return synth.build_case("costs", nx, ny, synth.uniform_layers(nz, 5.0 * nz), **d)


def times(case, precision, nsteps=8):
    """Device time (ms) of a resident step, its advection and its column kernel."""
    import torch
    t = gpu.TracerStep(case, precision=precision)
    t.start()
    t.run(4)
    t.sync()
    s = torch.cuda.ExternalStream(t.stream())
    best = np.inf
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(s)
        t.run(nsteps)
        b.record(s)
        b.synchronize()
        best = min(best, a.elapsed_time(b) / nsteps)
    t.profile(True)
    t.run(nsteps)
    t.sync()
    adv, col = t.kernel_time(1)[0], t.kernel_time(2)[0]
    t.close()
    return best, adv, col


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP32_COMP])
def test_set_up_of_few_layers(precision):
    """Two layers: the step beside its transport kernels 0.16 of them (0.56 where
    a block has eight warps whatever the layers)."""
    step, adv, col = times(window(1000, 800, 2, 3), precision)
    assert step - adv - col < 0.35 * (adv + col)


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP32_COMP, gpu.FP64])
@pytest.mark.parametrize("nz", [4, 8])
def test_column_kernel_default_in_shallow_columns(precision, nz):
    """The default number of warps per block is within 15 % of the best (it was 1.3
    to 1.8 times as slow where a block had as many as its memory holds)."""
    case = window(400, 300, nz, 16)
    t = gpu.TracerStep(case, precision=precision)
    t.start()
    t.run(3)
    t.sync()

    def col(warps):
        t.set_tiling(tracers=warps)
        best = np.inf
        for _ in range(3):
            t.profile(True)
            t.run(4)
            t.sync()
            best = min(best, t.kernel_time(2)[0])
        t.profile(False)
        return best

    default = col(t.get_tuning()["tracers_per_block"])
    rest = [col(w) for w in (2, 4, 8)]
    t.close()
    assert default <= 1.15 * min(rest)
