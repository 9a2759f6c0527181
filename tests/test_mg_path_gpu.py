"""Which multigrid cycle a case runs, in clusters of how many blocks, and phi
after a fixed number of cycles.

A mode's lines live in its cluster's shared memory wherever a cluster of at
most 16 blocks holds them; FITS gives the smallest that does, FP64 and mixed.
Modes that none holds, SOR modes and mixed spans finer than 1/11 run the cycle
in global memory.  Every mode takes CYCLES of them, the criterion being out of
reach, on the GPU and in the oracle, so the iterates are those of the same
cycle also in the mixed form, which at a criterion may stop one sooner or
later: 1e-10 relative in FP64, and 1e-5 in the mixed form, whose cycle carries
about fifty FP32 roundings (3e-6)."""
import ctypes as C

import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver
from test_mg_resident_gpu import SHAPES, build, divergence, solve

pytestmark = pytest.mark.gpu

FITS = {("x_ft", 48, 97): (2, 2), ("z_ft", 64, 129): (4, 4), ("duct", 32, 193): (4, 2), ("x_ft", 16, 256): (2, 1),
        ("x_ft", 128, 96): (4, 4)}


def path(s):
    fn = s.lib.lesgpu_check_mg
    fn.argtypes = [C.c_void_p, C.POINTER(C.c_int64), C.POINTER(C.c_int64)]
    resident, blocks = C.c_int64(), C.c_int64()
    assert fn(s.h, C.byref(resident), C.byref(blocks)) == 0
    return resident.value, blocks.value


CYCLES = 6


def fixed(c, **kw):
    c.settings = dict(c.settings, resid1=1e-300, mgitr=CYCLES, **kw)
    return c


def check_phi(oracle_lib, c, tol, s):
    d = divergence(c.grid)
    got, _ = solve(s, d)
    ref = cases.Case(c.name, dict(c.settings, precision=abi.PREC_FP64), c.grid, c.grid_dat, c.grid_bin, c.fields,
                     time=c.time, dt=c.dt, ibm=c.ibm)
    want, _ = solve(solver.Solver(oracle_lib, "ref_", ref), d)
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("flow,nl,n2m,nlev", SHAPES)
def test_resident(oracle_lib, monkeypatch, flow, nl, n2m, nlev):
    monkeypatch.setenv("LESGPU_AUTOTUNE", "0")
    least = FITS.get((flow, nl, n2m), (1, 1))
    for q, (prec, tol) in enumerate(((abi.PREC_FP64, 1e-10), (abi.PREC_MIXED, 1e-5))):
        for cap in (1, 2, 4, 8, 16):
            monkeypatch.setenv("LESGPU_MG_CLUSTER_MAX", str(cap))
            c = fixed(build(flow, nl, n2m, nlev, prec))
            s = leswht_gb300.gpu_solver(c)
            assert path(s) == (1, max(cap, least[q]))
            if cap in (1, 16):
                check_phi(oracle_lib, c, tol, s)
            s.close()


@pytest.mark.parametrize("n,nbli", [((256, 192, 2), None),      # no cluster holds a mode
                                    ((64, 48, 8), 80)])         # more half sweeps than a schedule takes
def test_global_memory(oracle_lib, n, nbli):
    c = cases.cylinder(*n)
    c = fixed(c, nbli=nbli or c.settings["nbli"])
    s = leswht_gb300.gpu_solver(c)
    assert path(s)[0] == 0
    check_phi(oracle_lib, c, 1e-10, s)


def test_global_memory_fine_span(oracle_lib):
    """dz = 1/20 in the mixed form; the FP64 form of the case, and the mixed
    form at dz = 1/10, stay in the clusters."""
    c = fixed(cases.cylinder(32, 24, 64, precision=abi.PREC_MIXED))
    s = leswht_gb300.gpu_solver(c)
    assert path(s)[0] == 0
    check_phi(oracle_lib, c, 1e-5, s)
    assert path(leswht_gb300.gpu_solver(cases.cylinder(32, 24, 64)))[0] == 1
    assert path(leswht_gb300.gpu_solver(cases.cylinder(32, 24, 32, precision=abi.PREC_MIXED)))[0] == 1
