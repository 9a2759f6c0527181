"""A zero residual meets any positive criterion, also one whose square
underflows: without a right-hand side the first norm test stops every mode,
as sqrt(0) < test does in the oracle.  A criterion of zero is never met."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver
from test_mg_resident_gpu import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("resid1", [1e-6, 1e-150, 1e-160, 1e-170, 1e-300, 0.0])
def test_no_right_hand_side(oracle_lib, monkeypatch, resid1, prec):
    monkeypatch.setenv("LESGPU_AUTOTUNE", "0")
    def case(p):
        c = cases.cylinder(16, 24, 4, nlev=2, precision=p)
        c.settings = dict(c.settings, resid1=resid1, mgitr=5)
        return c
    zero = np.zeros(case(prec).grid.shape)
    ref = solver.Solver(oracle_lib, "ref_", case(abi.PREC_FP64))
    want, iters = solve(ref, zero)
    s = leswht_gb300.gpu_solver(case(prec))
    got, n = solve(s, zero)
    assert n == iters
    assert s.report()["poisson_unconverged"] == ref.report()["poisson_unconverged"] == (0 if resid1 > 0.0 else 3)
    assert not got.any() and not want.any()
