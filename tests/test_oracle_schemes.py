"""The CPU oracle's ORDER1, ORDER2, ORDER4, QUICKEST_CO and ORDER2_UW against the
reference's own tracer step (tests/golden; CPU only), bit for bit."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))

import oracle  # noqa: E402
from cases import SCHEME_CASES, build, input_digest  # noqa: E402


@pytest.mark.parametrize("name", sorted(SCHEME_CASES))
def test_oracle_matches_reference_fixture(name):
    case, nsteps = build(name)
    g = np.load(os.path.join(HERE, "golden", name + ".npz"))
    rc, tr, sur, nsur, d = oracle.run_oracle(case, nsteps)
    assert rc == int(g["status"])
    np.testing.assert_array_equal(sur, g["sur_t"])
    np.testing.assert_array_equal(nsur, g["nsur_t"])
    assert d.nwarn == int(g["nwarn"])
    if input_digest(case) == str(g["digest"]):
        np.testing.assert_array_equal(tr, g["tr"])
    else:
        cells = np.arange(1, case.win.sgsiz)
        assert oracle.max_rel_err(tr, g["tr"], cells).max() <= 1e-12
