"""The step's volume sums against numpy over the fields it left: flow rate,
temperature volume, bulk velocity and temperature, wall-shear sums, divergence
and eddy-viscosity maxima, from boxes of a few blocks to ones whose threads
take whole and part groups of cells.  A sum is at most ~40
rounded additions deep on the device and its weights three products, so
1e-14 of the sum of magnitudes."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases

pytestmark = pytest.mark.gpu

TOL = 1e-14


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("n", [(8, 9, 8), (30, 33, 24), (64, 64, 75), (64, 64, 80), (128, 64, 75), (128, 64, 80)])
def test_sums(n, prec):
    c = cases.channel(*n, precision=prec)
    s = leswht_gb300.gpu_solver(c)
    for _ in range(2):
        r = s.step()
    f, g = s.fields(), c.grid
    n1, n2, n3 = n
    I = np.s_[1:n3 + 1, 1:n2 + 1, 1:n1 + 1]
    w = lambda a, b, d: d[1:n3 + 1, None, None] * b[None, 1:n2 + 1, None] * a[None, None, 1:n1 + 1]
    A = {k: np.asarray(getattr(g, k)) for k in ("f2fx", "f2fy", "f2fz", "c2cx", "f2fxi", "f2fyi", "f2fzi", "c2cyi")}
    cu, cc = w(A["c2cx"], A["f2fy"], A["f2fz"]), w(A["f2fx"], A["f2fy"], A["f2fz"])
    u, t = f["u"][I], f["t"][I]

    def near(x, terms, scale=1.0):
        assert abs(x - terms.sum() / scale) <= TOL * np.abs(terms).sum() / scale

    near(r["qvol"][0], u * cu)
    near(r["tvol"][2], t * cc)
    near(r["tvol"][0], t * cc)
    near(r["ubulk"], u * cu, cu.sum())
    near(r["tbulk_fluid"], t * cu, cu.sum())
    dv = np.abs(np.diff(f["u"][1:n3 + 1, 1:n2 + 1, 1:n1 + 2], axis=2) * A["f2fxi"][None, None, 1:n1 + 1]
                + np.diff(f["v"][1:n3 + 1, 1:n2 + 2, 1:n1 + 1], axis=1) * A["f2fyi"][None, 1:n2 + 1, None]
                + np.diff(f["w"][1:n3 + 2, 1:n2 + 1, 1:n1 + 1], axis=0) * A["f2fzi"][1:n3 + 1, None, None])
    mag = sum(2.0 * np.abs(f[k]).max() * A[d].max() for k, d in (("u", "f2fxi"), ("v", "f2fyi"), ("w", "f2fzi")))
    assert abs(r["dvmax"] - dv.max()) <= 1e-15 * mag           # four roundings of each side's terms
    area = A["c2cx"][None, 1:n1 + 1] * A["f2fz"][1:n3 + 1, None]
    re, vol = c.settings["re"], g.xl * g.yl * g.zl
    for q, (j, jn, a, b) in ((1, (1, 2, 1, 2)), (2, (n2, n2 - 1, n2 + 1, n2))):
        d1 = 1.0 / A["c2cyi"][a]
        d2 = d1 + 1.0 / A["c2cyi"][b]
        k = area / (d1 * d2 * (d2 - d1) * re * vol)
        x, y = f["u"][1:n3 + 1, j, 1:n1 + 1] * d2 * d2 * k, f["u"][1:n3 + 1, jn, 1:n1 + 1] * d1 * d1 * k
        assert abs(r["pmi"][q] - (x - y).sum()) <= TOL * (np.abs(x) + np.abs(y)).sum()
    nut = s.get(abi.F_NUSGS)[I]
    near(r["nutavg"], nut * cc * re, cc.sum())
    assert r["nutmax"] == pytest.approx(max(nut.max(), 0.0) * re, rel=1e-15)
