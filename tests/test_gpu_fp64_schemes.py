"""Every FP64 scheme where the advection kernel's warps climb several layers, at the
edges of its tiles, across moving surfaces and at the ends of the range, bitwise
against the oracle.

A warp climbs a chunk of layers, the longest that leaves about six rounds of warps:
one layer in small windows, so the windows here are large enough for two and more.
A chunk's first layer works out its bottom flux, the others take the flux kept from
the layer below.  Tolerance: none.
"""
import numpy as np
import pytest

import oracle
from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]

SCHEMES = {"quickest": 0x20, "vanleer": 0x80, "order1": 0x2, "order2": 0x4, "order4": 0x10,
           "quickest_co": 0x40, "order2_uw": 0x2000}
NEW = ["order1", "order2", "order4", "quickest_co", "order2_uw"]
LAYERS = np.array([-30.0, -22.0, -14.0, -8.0, -3.0, -1.0, 0.6, 2.5])


def window(nx, ny, nz, ntr, scheme, **kw):
    d = dict(seed=91, ntr=ntr, depth=(3.0, 5.0 * nz - 1.0), land_frac=0.15, cell=(400.0, 900.0),
             curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1), tracers=("logn", 1e-2, 10.0),
             trasc=SCHEMES[scheme], ultimate=int(scheme != "order1"))
    d.update(kw)
    layers = d.pop("layers", synth.uniform_layers(nz, 5.0 * nz))
    return synth.build_case("schemes", nx, ny, layers, **d)


def check(case, nsteps=2):
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


# columns of 1 to 61 layers: chunks of 2 (230 x 190) and 3 layers (265 x 220), which do
# not divide the columns' layers, floors anywhere in a chunk
@pytest.mark.parametrize("nx,ny", [(230, 190), (265, 220)])
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
def test_climb(scheme, nx, ny):
    check(window(nx, ny, 61, 2, scheme), nsteps=1)


@pytest.mark.parametrize("scheme", ["quickest", "vanleer", "order4", "order2_uw"])
def test_climb_with_horizontal_diffusion_and_mixed_flags(scheme):
    """One tracer only diffuses, one only advects, one does both."""
    case = window(230, 190, 61, 3, scheme, hdiff=(40.0, [1, 0, 1]))
    arrays = case.opts_arrays()
    arrays["advect"] = np.array([0, 1, 1], np.int32)
    case.opts_arrays = lambda: arrays
    check(case, nsteps=1)


@pytest.mark.parametrize("scheme", ["quickest", "vanleer", "order1", "order4"])
def test_climb_across_a_moving_surface(scheme):
    """Open floors as well, and surfaces that move through two layer faces."""
    layers = np.concatenate([np.linspace(-290.0, -3.0, 59), [-1.0, 0.6, 2.5]])
    case = window(230, 190, 61, 2, scheme, layers=layers, depth=(4.0, 289.0),
                  eta_offset=(1.9, -1.7))
    case.w[case.win.bot_t[1:case.win.ncol + 1][::5]] = 2e-6
    check(case)


@pytest.mark.parametrize("scheme", ["quickest", "order4"])
def test_climb_of_more_tracers_than_a_row(scheme):
    """70 tracers: three groups, chunks of 2 layers."""
    check(window(100, 90, 41, 70, scheme, depth=(150.0, 204.0)), nsteps=1)


@pytest.mark.parametrize("scheme", ["quickest", "order2"])
def test_climb_of_whole_columns(scheme):
    """A chunk is a column of three layers."""
    check(window(760, 700, 3, 1, scheme, land_frac=0.0, depth=(14.0, 14.9)), nsteps=1)


@pytest.mark.parametrize("nx,ny,nz,ntr", [(31, 9, 7, 2), (33, 9, 7, 2), (64, 5, 9, 1),
                                          (9, 40, 40, 5), (40, 12, 5, 70)])
@pytest.mark.parametrize("scheme", NEW)
def test_sizes(scheme, nx, ny, nz, ntr):
    check(window(nx, ny, nz, ntr, scheme), nsteps=3)


@pytest.mark.parametrize("ntr", [2, 5, 9])
def test_column_kernel_of_128_layers(ntr):
    """Shared memory for fewer warps than tracers."""
    check(window(97, 6, 128, ntr, "quickest", depth=(500.0, 639.0)), nsteps=3)


@pytest.mark.parametrize("scheme", NEW)
@pytest.mark.parametrize("hdiff", [None, (40.0, [1, 0, 1])])
def test_crossing_surface(scheme, hdiff):
    """The surface moves through layer faces at -1.0 and 0.6 m."""
    check(window(45, 20, 7, 3, scheme, layers=LAYERS, depth=(4.0, 29.0), eta_offset=(1.9, -1.7),
                 hdiff=hdiff), nsteps=4)


@pytest.mark.parametrize("scale", [1e-308, 1e-290, 1e-160, 1e-120, 1e120, 1e160, 1e290])
@pytest.mark.parametrize("scheme", sorted(set(SCHEMES) - {"quickest"}))
def test_extreme_values(scheme, scale):
    """Every other tracer holds zeros, equal neighbours and sign changes too."""
    case = window(40, 12, 6, 4, scheme)
    c = case.win.wet_cells()
    case.tr *= scale
    case.tr[1, c[::3]] = 0.0
    case.tr[2, c] = np.where(c % 5 < 2, -case.tr[2, c], case.tr[2, c])
    case.tr[3, c] = scale * (c % 2)
    check(case, nsteps=3)
