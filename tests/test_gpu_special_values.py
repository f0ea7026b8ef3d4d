"""FP64 tracers that are negative zeros, infinities, NaN or near the ends of the
range, against the oracle: the same bits where the oracle has a number, NaN
where it has NaN.
"""
import numpy as np
import pytest

import oracle
from ems_b200 import _abi, gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]

SCHEMES = {"quickest": 0x20, "vanleer": 0x80, "order1": 0x2, "order2": 0x4, "order4": 0x10,
           "quickest_co": 0x40, "order2_uw": 0x2000}
ENAN = 3


def window(scheme, ultimate, vdiff, ntr=4, **kw):
    d = dict(seed=11, ntr=ntr, depth=(3.0, 39.0), land_frac=0.15, cell=(400.0, 900.0),
             curvilinear=True, umax=0.8, kz=("logu", 1e-5, 1e-1), tracers=("logn", 1e-2, 10.0),
             trasc=SCHEMES[scheme], ultimate=ultimate)
    d.update(kw)
    case = synth.build_case("special", 36, 15, synth.uniform_layers(8, 40.0), **d)
    if not vdiff:  # the implicit solve turns -0 into 0 and spreads a NaN over its column
        arrays = case.opts_arrays()
        arrays["tdif_v"] = arrays["tdif_v"][:0]
        case.opts_arrays = lambda: arrays
    return case


def check(case, nsteps=1):
    t = gpu.TracerStep(case)
    t.start()
    t.run(nsteps)
    rc = 0
    try:
        t.sync()
    except _abi.StatusError as e:
        rc = e.code
    tr = t.download()
    t.close()
    orc, ref, *_ = oracle.run_oracle(case, nsteps)
    assert rc == orc and rc in (0, ENAN)
    c = case.win.wet_cells()
    a, b = tr[:, c], ref[:, c]
    np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    ok = ~np.isnan(b)
    np.testing.assert_array_equal(a[ok].view(np.int64), b[ok].view(np.int64))
    return b


ALL = [(s, u) for s in sorted(SCHEMES) for u in (0, 1) if not (s == "order1" and u)]


@pytest.mark.parametrize("scheme,ultimate", ALL)
def test_negative_zeros(scheme, ultimate):
    """Still water of both zeros, and drops of either sign in it."""
    case = window(scheme, ultimate, vdiff=False)
    c = case.win.wet_cells()
    r = np.random.default_rng(3)
    case.tr[:, c] = np.where(r.random((4, len(c))) < 0.5, 0.0, -0.0)
    case.tr[0, c] = -0.0
    drops = r.random((4, len(c))) < 0.05
    drops[:2] = False
    case.tr[:, c] = np.where(drops, r.normal(size=(4, len(c))), case.tr[:, c])
    ref = check(case)
    assert np.any(ref == 0.0)


@pytest.mark.parametrize("scheme,ultimate", ALL)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1.7e308])
def test_not_finite(scheme, ultimate, value):
    """Single cells that are not finite or too large to be added, some of them
    on the floor and in the layer above it."""
    case = window(scheme, ultimate, vdiff=False)
    w = case.win
    c = w.wet_cells()
    bots = w.bot_t[1:w.ncol + 1]
    case.tr[0, c[::97]] = value
    case.tr[1, bots[::31]] = value
    case.tr[2, w.zp1[bots[5::31]]] = value
    check(case)


@pytest.mark.parametrize("scheme,ultimate", ALL)
def test_not_finite_with_vertical_diffusion(scheme, ultimate):
    case = window(scheme, ultimate, vdiff=True)
    w = case.win
    case.tr[0, w.bot_t[1:w.ncol + 1][::31]] = np.inf
    case.tr[1, w.wet_cells()[::97]] = np.nan
    check(case)
