"""What the host side of a call touches and waits for."""
import numpy as np
import pytest

from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


def test_set_preamble_does_not_wait_for_the_default_stream():
    """A forecast sets the preamble each step; only the first call has arrays to
    fill, so a later one returns while the caller's own kernels still run."""
    import torch
    case = synth.make("small")
    t = gpu.TracerStep(case)
    t.start()
    t.set_preamble(True)
    t.run(1)
    t.sync()
    torch.cuda._sleep(1000)  # loads the kernel
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(int(1e9))  # about half a second on the default stream
    done.record()
    t.set_preamble(True, np.zeros(case.win.sgsizS))
    assert not done.query()
    torch.cuda.synchronize()
    t.run(1)
    t.sync()
    t.close()
