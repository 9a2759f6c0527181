"""poiss_mgrd's line solves (half a warp per y line, its rows in the lanes'
registers) on every length class and remainder and with odd numbers of lines,
levels that run on block 0 alone and levels that do not, and lines too long
for the registers, against the CPU oracle: phi after a fixed number of
iterations to 1e-10 relative, the bound of the other poiss_mgrd tests.  Lines
of more than 100 rows, stretched over a few wide cells in x and z, get 1e-6:
their LU factors alone carry 4e-13 to 1.4e-12 (against 80-bit arithmetic, the
serial recurrence and the scan alike) and the iteration magnifies that by up
to 1e5, on any order of operations."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver

pytestmark = pytest.mark.gpu

# (n1, n2, n3, nlev, walls in z)
SHAPES = [(8, 17, 8, 1, False), (16, 33, 8, 2, False), (16, 50, 16, 0, False), (12, 64, 6, 1, True), (32, 65, 16, 3, False),
          (10, 90, 4, 0, False), (16, 97, 16, 2, True), (8, 129, 8, 2, False), (8, 200, 8, 1, False), (4, 256, 4, 1, False),
          (8, 258, 4, 1, False)]


@pytest.mark.parametrize("n1,n2,n3,nlev,walls", SHAPES)
def test_fixed_iterations_match_the_oracle(oracle_lib, n1, n2, n3, nlev, walls):
    c = cases.with_poisson(cases.channel(n1, n2, n3, zwalls=walls), abi.POISSON_MGRD, nlev=nlev)
    c.settings.update(mgitr=2, resid1=1e-30)
    g, r = leswht_gb300.gpu_solver(c), solver.Solver(oracle_lib, "ref_", c)
    for s in (g, r):
        s.phase(abi.PH_STEPINIT)
        s.phase(abi.PH_SUBSTEPINIT, 1)
    r.phase(abi.PH_SGS, 1)
    r.phase(abi.PH_RHSNLHS, 1)
    r.phase(abi.PH_DIVGS, 1)
    g.set(abi.F_DIVGSUM, r.get(abi.F_DIVGSUM))
    for s in (g, r):
        s.phase(abi.PH_POISSON, 1)
    a, b = g.get(abi.F_PHI), r.get(abi.F_PHI)
    assert np.linalg.norm(a - b) <= (1e-10 if n2 <= 100 else 1e-6) * np.linalg.norm(b)
