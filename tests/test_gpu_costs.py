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
@pytest.mark.parametrize("nx,ny,nz,ntr", [(400, 300, 4, 16), (400, 300, 8, 16), (46, 139, 9, 24),
                                          (152, 20, 35, 5), (252, 21, 16, 18)])
def test_column_kernel_default_in_shallow_columns(precision, nx, ny, nz, ntr):
    """The default number of warps per block is within 20 % of the best.  In large
    windows of few layers it was 1.3 to 1.8 times as slow where a block had as many
    as its memory holds; where there are fewer tiles than SMs it is 1.4 to 1.8 times
    as slow with as few as those take."""
    case = window(nx, ny, nz, ntr)
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
    assert default <= 1.2 * min(rest)


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP32_COMP, gpu.FP64])
def test_column_kernel_where_no_column_has_all_layers(precision):
    """60 layers, columns of 8 at most, one tracer: the column kernel takes what it
    takes in a window of 8 layers (2.5 to 3.5 times that where its shared memory
    is sized for 60)."""
    shallow = times(window(400, 300, 60, 1, depth=(3.0, 39.0)), precision)
    few = times(window(400, 300, 8, 1, depth=(3.0, 39.0)), precision)
    assert shallow[2] < 1.5 * few[2]


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP32_COMP, gpu.FP64])
def test_column_kernel_with_a_trench(precision):
    """128 layers on a few columns, 18 at most on the others, one tracer: the
    column kernel takes four times what it takes without them (6.7 where the
    shallow tiles run at the deep ones' few blocks an SM)."""
    layers = synth.uniform_layers(128, 640.0)
    r = np.random.default_rng(5)
    bathy = -5.0 * r.uniform(2.0, 18.0, (200, 300))
    land = np.zeros((200, 300), np.uint8)
    flat = window(300, 200, 128, 1, bathy_land=(synth._snap_bathy(bathy, layers), land))
    bathy[:, :9] = -639.0
    trench = window(300, 200, 128, 1, bathy_land=(synth._snap_bathy(bathy, layers), land))
    assert times(trench, precision)[2] < 5.2 * times(flat, precision)[2]


@pytest.mark.parametrize("precision", [gpu.FP32_MIXED, gpu.FP64])
def test_set_up_where_no_column_has_all_layers(precision):
    """128 layers, columns of 20 at most: the step beside its transport kernels takes
    about what it takes in a window of 20 layers (twice that with shared memory
    for 128)."""
    a, b = (times(window(300, 200, nz, 1, depth=(3.0, 99.0)), precision) for nz in (128, 20))
    assert a[0] - a[1] - a[2] < 1.5 * (b[0] - b[1] - b[2])


def test_fp64_advection_where_no_column_has_all_layers():
    """60 layers, columns of 8 at most: the FP64 advection kernel takes what it takes
    in a window of 8 layers (1.4 times that where its chunks of layers are counted
    over 60)."""
    a, b = (times(window(400, 300, nz, 1, depth=(3.0, 39.0)), gpu.FP64) for nz in (60, 8))
    assert a[1] < 1.2 * b[1]


def test_column_kernel_of_any_depth_stays_one_launch():
    """128 layers, columns of any depth, three tracers: too few tiles for more
    launches than one (three took 1.4 times as long as one).  Launches are counted:
    k_adv32, k_vd32 and k_general of a sub-step, k_lateral and k_set_dz."""
    t = gpu.TracerStep(window(150, 120, 128, 3), precision=gpu.FP32_MIXED)
    t.start()
    t.run(3)
    t.sync()
    n = t.launches()
    t.run(4)
    t.sync()
    assert t.launches() - n == 4 * 5
    t.close()
