"""The FP64 stencils with 1-D weights and the plane-marching test filter against
the oracle: walls, wrapped and ghost neighbours in each direction, every test
filter (x, z, both), plane counts that leave a filter run part empty down to a
single plane, without and with the temperature decomposition.  Bound: the
step's parity bound, 1e-10 of each field's norm."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver

pytestmark = pytest.mark.gpu


def duct(n1, n2, n3):
    return cases.with_poisson(cases.channel(n1, n2, n3, zwalls=True), abi.POISSON_X_FT, nlev=1)


@pytest.mark.parametrize("build,n,settings", [
    (cases.channel, (12, 10, 9), dict(filter=3)),
    (cases.channel, (10, 9, 15), dict(filter=1)),
    (cases.channel, (16, 8, 3), dict(filter=2)),
    (cases.channel, (40, 33, 60), dict(filter=3)),
    (cases.channel, (12, 10, 8), dict(filter=3, gr=50.0, grdir=1)),
    (cases.channel, (12, 10, 8), dict(filter=3, idecomp=0, gr=50.0, grdir=2)),
    (duct, (12, 14, 10), dict(filter=3)),
    (cases.cylinder, (44, 36, 6), dict(filter=3, gr=50.0, grdir=3)),
])
def test_two_steps(oracle_lib, build, n, settings):
    case = build(*n)
    case.settings.update(settings)
    g, r = leswht_gb300.gpu_solver(case), solver.Solver(oracle_lib, "ref_", case)
    for _ in range(2):
        g.step(); r.step()
    fg, fr = g.fields(), r.fields()
    s = np.s_[1:n[2] + 1, 1:n[1] + 1, 1:n[0] + 1]
    for f, name in ((abi.F_NUSGS, "nusgs"), (abi.F_ALSGS, "alsgs")):
        fg[name], fr[name] = g.get(f)[s], r.get(f)[s]
    for k in fr:
        assert np.linalg.norm(fg[k] - fr[k]) <= 1e-10 * max(np.linalg.norm(fr[k]), 1e-300), k
