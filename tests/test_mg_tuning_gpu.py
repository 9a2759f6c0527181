"""The multigrid's tuned cluster sizes are kept by shape, form and cycle: the
second form of a shape starts and solves, whichever form tuned first.

64x64 modes: in FP32 one block holds a mode, in FP64 none of fewer than two
does, so under a cap of one block the forms take different sizes.  224x150
modes: in FP32 16 blocks hold one; in FP64 none do and the cycle in global
memory runs, whose levels 16 blocks do not split evenly.  phi of the FP64 form
as in the other multigrid tests, 1e-10 of the oracle's; the mixed form's 1e-5
where both take the same cycles."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver
from test_mg_resident_gpu import divergence, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap,first", [((64, 64, 4), "1", "mixed"), ((64, 64, 6), "1", "fp64"),
                                         ((224, 150, 4), None, "mixed"), ((224, 150, 6), None, "fp64")])
def test_forms_of_one_shape(oracle_lib, monkeypatch, n, cap, first):
    monkeypatch.setenv("LESGPU_AUTOTUNE", "1")
    if cap:
        monkeypatch.setenv("LESGPU_MG_CLUSTER_MAX", cap)
    form = {"mixed": abi.PREC_MIXED, "fp64": abi.PREC_FP64}
    case = {f: cases.cylinder(*n, precision=p) for f, p in form.items()}
    d = divergence(case["fp64"].grid)
    want, iters = solve(solver.Solver(oracle_lib, "ref_", case["fp64"]), d)
    for f in (first, "fp64" if first == "mixed" else "mixed"):
        s = leswht_gb300.gpu_solver(case[f])
        got, k = solve(s, d)
        if f == "fp64":
            assert k == iters
        assert abs(k - iters) <= 1
        if k == iters:
            assert np.linalg.norm(got - want) <= (1e-10 if f == "fp64" else 1e-5) * np.linalg.norm(want)
        s.close()
