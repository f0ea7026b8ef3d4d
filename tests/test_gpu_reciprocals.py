"""FP64 quotients formed from reciprocals, bitwise against the oracle where they
are hardest: a divisor whose significand is all ones (2 - 2^-52 times a power
of two), whose Newton reciprocal ends on a tie, under a power of two.

Tolerance: none, the results are the reference's bits.
"""
import numpy as np
import pytest

import oracle
from ems_b200 import gpu, synth

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("need_gpu")]

ONES = 2.0 - 2.0 ** -52
SCHEMES = {"quickest": 0x20, "vanleer": 0x80, "order2": 0x4, "order4": 0x10,
           "quickest_co": 0x40, "order2_uw": 0x2000}


@pytest.mark.parametrize("scale", [0, -37, 200])
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
def test_all_ones_divisors(scheme, scale):
    """The limiter's td - tu is 2 - 2^-52 and tc - tu a power of two, at small
    and at capped Courant numbers, for flow of either sign."""
    case = synth.build_case(
        "ones", 60, 40, synth.uniform_layers(8, 40.0), seed=5, ntr=6, depth=(20.0, 39.0),
        land_frac=0.1, cell=(400.0, 900.0), curvilinear=True, umax=0.8, dt=200.0,
        kz=("logu", 1e-5, 1e-1), trasc=SCHEMES[scheme], ultimate=1)
    w = case.win
    c = w.wet_cells()
    r = np.random.default_rng(7)
    for n in range(case.ntr):
        # tracers 0-1 vary along i, 2-3 along j, 4-5 in every direction; half of
        # the cells 0, so that tu is; the rest the divisor or a power of two
        key = (w.s2i[c], w.s2j[c], np.arange(len(c)))[n // 2]
        m = key.max() + 1
        kind = r.integers(0, 4, m)
        v = np.where(kind < 2, 0.0, np.where(kind == 2, ONES, np.ldexp(1.0, r.integers(-15, 4, m))))
        case.tr[n, c] = (1 - 2 * (n & 1)) * v[key] * 2.0 ** scale
    t = gpu.TracerStep(case)
    t.start()
    t.run(1)
    t.sync()
    tr = t.download()
    t.close()
    rc, ref, *_ = oracle.run_oracle(case, 1)
    assert rc == 0
    np.testing.assert_array_equal(tr[:, 1:], ref[:, 1:])
