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
