"""The multigrid cycles that keep a mode in its cluster's shared memory
(k_mgl.cuh) on lines of every length class and remainder, and on every
cluster size that holds the mode, against the CPU oracle.

FP64: the same cycle counts and phi to 1e-10 relative, the parity bound of the
other Poisson tests.  Mixed form: the same FP64 residual test stops it, a cycle
sooner or later where its FP32 corrections differ at the criterion; a cycle's
correction carries about fifty FP32 roundings (3e-6 relative) and what it
leaves is taken up by the cycles after it, so phi matches the oracle's to 1e-5
relative when both take the same cycles."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver

pytestmark = pytest.mark.gpu


def build(flow, nl, n2m, nlev, prec):
    if flow == "z_ft":
        c = cases.cylinder(nl, n2m, 4, nlev=nlev, precision=prec)
    else:
        c = cases.with_poisson(cases.channel(8, n2m, nl, zwalls=flow == "duct", precision=prec), abi.POISSON_X_FT, nlev=nlev)
    return c


def divergence(g):
    """Seeded noise without a net source."""
    d = np.random.default_rng(11).standard_normal((g.n3m, g.n2m, g.n1m))
    w = (g.f2fz[1:g.n3m + 1, None, None] * g.f2fy[None, 1:g.n2m + 1, None] * g.f2fx[None, None, 1:g.n1m + 1])
    out = np.zeros(g.shape)
    out[1:g.n3m + 1, 1:g.n2m + 1, 1:g.n1m + 1] = d - (d * w).sum() / w.sum()
    return out


def solve(s, d):
    s.phase(abi.PH_STEPINIT)
    s.phase(abi.PH_SUBSTEPINIT, 1)
    s.set(abi.F_DIVGSUM, d)
    s.phase(abi.PH_POISSON, 1)
    return s.get(abi.F_PHI), s.report()["poisson_iters"][0]


# line lengths around the classes of 2, 3, 4, 6, 8, 12 and 16 rows a lane;
# line counts with even, odd and non-power-of-two pair counts; one level to six
SHAPES = [("z_ft", 64, 48, 5), ("z_ft", 32, 33, 3), ("duct", 16, 17, 3), ("duct", 48, 50, 4), ("x_ft", 24, 64, 2),
          ("x_ft", 32, 65, 4), ("duct", 8, 90, 1), ("x_ft", 48, 97, 3), ("z_ft", 64, 129, 4), ("duct", 32, 193, 4),
          ("x_ft", 16, 256, 3), ("x_ft", 128, 96, 6)]


@pytest.mark.parametrize("flow,nl,n2m,nlev", SHAPES)
def test_cluster_sizes_match_the_oracle(oracle_lib, monkeypatch, flow, nl, n2m, nlev):
    monkeypatch.setenv("LESGPU_AUTOTUNE", "0")
    c = build(flow, nl, n2m, nlev, abi.PREC_FP64)
    d = divergence(c.grid)
    want, iters = solve(solver.Solver(oracle_lib, "ref_", c), d)
    assert 1 <= iters < c.settings["mgitr"]
    mixed = build(flow, nl, n2m, nlev, abi.PREC_MIXED)
    for cap in (1, 2, 4, 8, 16):
        monkeypatch.setenv("LESGPU_MG_CLUSTER_MAX", str(cap))
        got, n = solve(leswht_gb300.gpu_solver(c), d)
        assert n == iters, cap
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want), cap
        got, n = solve(leswht_gb300.gpu_solver(mixed), d)
        assert abs(n - iters) <= 1, cap
        if n == iters:
            assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want), cap
