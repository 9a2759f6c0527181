"""The mixed form's dynamic coefficient against values recorded with the test
filter that formed a cell's three planes anew: the filter that marches planes
rounds its FP32 sums in the same order, fma(c2, r, fma(c0, l, c1 m)) in x and
z.  Another order moves the coefficient, and with it every eddy viscosity, by
1.5e-5 to 5.2e-5 in these cases.  What else differs between the two are the
FP64 sums over the cells, within 1e-12."""
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases

pytestmark = pytest.mark.gpu

M = abi.PREC_MIXED


@pytest.mark.parametrize("build,csgsts", [
    (lambda: cases.with_poisson(cases.channel(32, 33, 32, amp=0.1, zwalls=True, precision=M), abi.POISSON_X_FT, nlev=3),
     7.414394242495127e-05),
    (lambda: cases.cylinder(64, 48, 8, re=3900.0, amp=0.05, precision=M), 0.0031645350821582277),
    (lambda: cases.cylinder_array(48, 40, 8, precision=M), 0.010331122409057222)])
def test_dynamic_coefficient(build, csgsts):
    s = leswht_gb300.gpu_solver(build())
    for ph in (abi.PH_STEPINIT, abi.PH_STEPINIT, abi.PH_SUBSTEPINIT, abi.PH_SGS):    # the first step runs without SGS
        s.phase(ph, 1)
    assert s.report()["csgsts"] == pytest.approx(csgsts, rel=1e-10)
