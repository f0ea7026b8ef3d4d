"""Which columns the FP64 tile kernels step, by what a step costs: a column that
goes the general path costs several times as much.  The results are compared
with the oracle bit for bit.
"""
import numpy as np
import pytest

import oracle
from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


def window(**kw):
    d = dict(seed=91, ntr=6, depth=(140.0, 149.0), land_frac=0.0, cell=(400.0, 900.0),
             curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1), tracers=("logn", 1e-2, 10.0))
    d.update(kw)
    return synth.build_case("routes", 200, 180, synth.uniform_layers(30, 150.0), **d)


def step_time(case, nsteps=8):
    """Device time of a resident step (ms), best of five."""
    import torch
    t = gpu.TracerStep(case)
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
    t.close()
    return best


def check(case, nsteps=2):
    t = gpu.TracerStep(case)
    t.start()
    t.run(nsteps)
    t.sync()
    tr = t.download()
    t.close()
    rc, ref, *_ = oracle.run_oracle(case, nsteps)
    assert rc == 0
    np.testing.assert_array_equal(tr[:, 1:], ref[:, 1:])


def test_open_floors_stay_with_the_tile_kernels():
    case = window()
    closed = step_time(case)
    case.w[case.win.bot_t[1:case.win.ncol + 1][::3]] = 2e-6
    assert step_time(case) < 1.5 * closed
    check(case)


def swap_east(case, i, j, k):
    """The east neighbours of two cells of one layer, in rows j and j + 1, swapped."""
    w = case.win
    a = next(c for c in w.wet_cells() if w.s2k[c] == k and w.s2i[c] == i and w.s2j[c] == j)
    b = w.yp1[a]
    ea, eb = int(w.xp1[a]), int(w.xp1[b])
    w.xp1[a], w.xp1[b], w.xm1[ea], w.xm1[eb] = eb, ea, b, a


def test_maps_that_do_not_stack_stay_with_the_tile_kernels():
    case = window()
    stacked = step_time(case)
    swap_east(case, 90, 40, 3)
    assert step_time(case) < 1.5 * stacked
    check(case)


@pytest.mark.parametrize("scheme,ultimate", [(0x20, 1), (0x20, 0), (0x80, 1), (0x2, 0), (0x4, 1),
                                             (0x10, 1), (0x40, 1), (0x2000, 0)])
@pytest.mark.parametrize("hdiff", [None, (40.0, [1, 0, 1])])
def test_maps_that_do_not_stack(scheme, ultimate, hdiff):
    """Every scheme, with and without horizontal diffusion: swapped cells in a
    warp's first, middle and last lanes, at the floor and at the surface."""
    case = synth.build_case(
        "swap", 34, 12, synth.uniform_layers(6, 30.0), seed=92, ntr=3, depth=(28.0, 29.0),
        cell=(400.0, 900.0), curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1),
        tracers=("logn", 1e-2, 10.0), trasc=scheme, ultimate=ultimate, hdiff=hdiff)
    for i, j, k in [(0, 1, 0), (9, 2, 3), (9, 4, 5), (30, 5, 2), (31, 7, 2), (14, 9, 5)]:
        swap_east(case, i, j, k)
    check(case)
