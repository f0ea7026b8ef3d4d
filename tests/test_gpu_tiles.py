"""The FP64 kernels at the edges of their tiles, bitwise against the oracle.

A warp of the advection kernel holds up to 32 neighbouring columns (the last
one only lending its west flux) and a chunk of layers; the column kernel 32
columns of one tracer.  Windows just below, at and above those sizes, one
tracer to more than a launch row of them, one layer to many, and tracers whose
values leave the range in which quotients are formed from reciprocals and the
limiter's cases from products.  Tolerance: none, the results are the
reference's bits.
"""
import numpy as np
import pytest

import oracle
from ems_b200 import _abi, gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]


def window(nx, ny, nz, ntr, **kw):
    d = dict(seed=91, ntr=ntr, depth=(3.0, 5.0 * nz - 1.0), land_frac=0.15, cell=(400.0, 900.0),
             curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1), tracers=("logn", 1e-2, 10.0))
    d.update(kw)
    layers = d.pop("layers", synth.uniform_layers(nz, 5.0 * nz))
    return synth.build_case("edge", nx, ny, layers, **d)


def check(case, nsteps=3):
    t = gpu.TracerStep(case)
    t.start()
    t.run(nsteps)
    t.sync()
    tr = t.download()
    sur, nsur = t.surface()
    t.close()
    rc, ref, rsur, rnsur, _ = oracle.run_oracle(case, nsteps)
    assert rc == 0
    np.testing.assert_array_equal(tr[:, 1:], ref[:, 1:])
    np.testing.assert_array_equal(sur, rsur)
    np.testing.assert_array_equal(nsur, rnsur)


@pytest.mark.parametrize("nx,ny,nz,ntr", [
    (30, 9, 7, 2), (31, 9, 7, 2), (32, 9, 7, 2), (33, 9, 7, 2), (63, 5, 2, 3), (64, 5, 9, 1),
    (9, 40, 40, 5), (97, 6, 128, 1), (40, 12, 5, 70)])
def test_sizes(nx, ny, nz, ntr):
    check(window(nx, ny, nz, ntr))


@pytest.mark.parametrize("scheme,ultimate", [(_abi.QUICKEST, 1), (_abi.QUICKEST, 0),
                                             (_abi.VANLEER, 1), (_abi.VANLEER, 0)])
@pytest.mark.parametrize("hdiff", [None, (40.0, [1, 0, 1])])
def test_crossing_surface(scheme, ultimate, hdiff):
    """The surface moves through layer faces at -1.0 and 0.6 m."""
    layers = np.array([-30.0, -22.0, -14.0, -8.0, -3.0, -1.0, 0.6, 2.5])
    check(window(45, 20, 7, 3, layers=layers, depth=(4.0, 29.0), eta_offset=(1.9, -1.7),
                 trasc=scheme, ultimate=ultimate, hdiff=hdiff), nsteps=4)


@pytest.mark.parametrize("scale", [1e-308, 1e-290, 1e-160, 1e-120, 1e120, 1e160, 1e290])
def test_extreme_values(scale):
    """Every other tracer holds zeros, equal neighbours and sign changes too."""
    case = window(40, 12, 6, 4)
    c = case.win.wet_cells()
    case.tr *= scale
    case.tr[1, c[::3]] = 0.0
    case.tr[2, c] = np.where(c % 5 < 2, -case.tr[2, c], case.tr[2, c])
    case.tr[3, c] = scale * (c % 2)
    check(case)


def test_open_floor():
    """Water through the floor: those columns go the general path."""
    case = window(50, 14, 8, 3)
    bots = case.win.bot_t[1:case.win.ncol + 1]
    case.w[bots[::3]] = 2e-6
    check(case)


def test_maps_that_do_not_stack():
    """East neighbours of one layer swapped between two rows: no column is a tile's."""
    case = window(20, 12, 6, 2, land_frac=0.0, depth=(28.0, 29.0))
    w = case.win
    wet = np.zeros(w.sgsiz, bool)
    wet[w.wet_cells()] = True
    a = next(c for c in w.wet_cells() if w.s2k[c] == 3 and w.s2i[c] == 9 and w.s2j[c] == 4)
    b = w.yp1[a]
    ea, eb = int(w.xp1[a]), int(w.xp1[b])
    assert wet[[a, b, ea, eb]].all()
    w.xp1[a], w.xp1[b], w.xm1[ea], w.xm1[eb] = eb, ea, b, a
    check(case)


@pytest.mark.parametrize("ntr", [12, 13, 31])
def test_dropin_chunks(ntr):
    """More than 2 MB of tracers cross the link in chunks: crossing surfaces and
    the thin-surface cursor, which runs through the tracers of a column."""
    layers = np.array([-30.0, -22.0, -14.0, -8.0, -3.0, -1.0, 0.6, 2.5])
    case = window(80, 60, 7, ntr, layers=layers, depth=(4.0, 29.0), eta_offset=(1.9, -1.7),
                  hmin=1.2, dt=1500.0)
    case.maxtr[:] = np.quantile(case.tr[0, case.win.wet_cells()], 0.6)
    assert case.tr.nbytes > 2 << 20
    tr, sur, nsur = case.copy_state()
    t = gpu.TracerStep(case)
    nsub = [t.step(tr, sur, nsur).nsub for _ in range(2)]
    t.close()
    assert max(nsub) > 1
    rc, ref, rsur, rnsur, _ = oracle.run_oracle(case, 2)
    assert rc == 0
    np.testing.assert_array_equal(tr[:, 1:], ref[:, 1:])
    np.testing.assert_array_equal(sur, rsur)
    np.testing.assert_array_equal(nsur, rnsur)


def test_more_tracers_than_an_fp32_launch_lists():
    """Compensated FP32: a tracer's values do not depend on how many there are."""
    def last(case, keep):
        t = gpu.TracerStep(case, precision=gpu.FP32_COMP)
        t.start()
        t.run(2)
        t.sync()
        tr = t.download()[keep]
        t.close()
        return tr[:, case.win.wet_cells()]
    many = window(33, 9, 7, 259)
    few = window(33, 9, 7, 4)
    keep = [0, 255, 256, 258]
    few.tr[:] = many.tr[keep]
    np.testing.assert_array_equal(last(many, keep), last(few, [0, 1, 2, 3]))


@pytest.mark.parametrize("nz", [3, 8, 9, 17, 33])
def test_preamble_depths(nz):
    """Columns shorter than, as long as and longer than a batch of cells, with
    surfaces that cross layer faces between the steps."""
    case = window(14, 11, nz, 2, eta_offset=(1.9, -1.7),
                  layers=np.concatenate([np.linspace(-5.0 * nz, -1.5, nz), [2.5]]))
    detadt = (case.eta - case.oldeta) / case.dt
    t = gpu.TracerStep(case)
    t.start()
    t.set_preamble(True, detadt)
    sur, nsur = case.sur_t.copy(), case.nsur_t.copy()
    for _ in range(2):
        want = oracle.preamble(case, detadt, sur, nsur)
        t.run(1)
        t.sync()
        got = t.get_flow()
        for k in ("w", "u1flux3d", "u2flux3d", "dzu1", "dzu2"):
            np.testing.assert_array_equal(got[k], want[k], err_msg=k)
        sur, nsur = t.surface()
    t.close()
