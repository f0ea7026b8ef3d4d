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


def test_dropin_reads_the_surface_vectors_from_element_one():
    """sur_t and nsur_t are 1-based: a caller may pass a pointer one element before
    its array, and what lies there may not be readable."""
    import ctypes as C
    import mmap
    from ems_b200 import _abi
    case = synth.make("small")
    n, page = case.win.ncol, mmap.PAGESIZE
    libc = C.CDLL(None, use_errno=True)
    libc.mprotect.argtypes = [C.c_void_p, C.c_size_t, C.c_int]
    tr, sur, nsur = case.copy_state()
    tr2 = tr.copy()
    keep, at = [], []
    for a in (sur, nsur):
        m = mmap.mmap(-1, page + -(-4 * n // page) * page)
        base = C.addressof(C.c_char.from_buffer(m))
        C.memmove(base + page, a.ctypes.data + 4, 4 * n)
        assert libc.mprotect(base, page, 0) == 0  # no access
        keep.append(m)
        at.append(base + page)
    t = gpu.TracerStep(case)
    st = case.make_state(tr, sur, nsur, keep)
    st.sur_t, st.nsur_t = [C.cast(p - 4, _abi.IP) for p in at]
    d = _abi.Diag()
    assert t.L.shoc_tr_gpu_step(t.h, C.byref(st), C.byref(d)) == 0
    t.step(tr2, sur, nsur)
    t.close()
    np.testing.assert_array_equal(tr[:, 1:], tr2[:, 1:])
    for p, a in zip(at, (sur, nsur)):
        np.testing.assert_array_equal(np.ctypeslib.as_array((C.c_int * n).from_address(p)), a[1:n + 1])
        assert libc.mprotect(p - page, page, 3) == 0
