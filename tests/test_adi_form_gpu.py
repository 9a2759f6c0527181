"""The form a sweep runs in is the one chosen for it.  Forms that cannot take a
batch give way to one thread a line, which a parity test does not notice."""
import ctypes as C

import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver
from test_adi_ends_gpu import CASES

pytestmark = pytest.mark.gpu


def other(s):
    fn = s.lib.lesgpu_check_adi_other
    fn.argtypes = [C.c_void_p, C.POINTER(C.c_int64)]
    n = C.c_int64(-1)
    assert fn(s.h, C.byref(n)) == 0
    return n.value


def two_ended(path, n, classes):
    path.write_text("".join(f"adi {n[0]} {n[1]} {n[2]} {d} {nc} 0 {per} {n[d]} 272\n" for d, nc, per in classes))


@pytest.mark.parametrize("q", range(len(CASES)))
def test_two_ended_runs(tmp_path, monkeypatch, q):
    _, build, (xper, zper) = CASES[q]
    case = build()
    two_ended(tmp_path / "tune.txt", (case.grid.n1m, case.grid.n2m, case.grid.n3m),
              [(d, nc, per) for d, per in ((0, xper), (1, 0), (2, zper)) for nc in (1, 3)])
    monkeypatch.setenv("LESGPU_AUTOTUNE", "1")
    monkeypatch.setenv("LESGPU_TUNE_FILE", str(tmp_path / "tune.txt"))
    s = leswht_gb300.gpu_solver(case)
    s.step()
    assert other(s) == 0


def test_conjugate_after_a_plain_case(oracle_lib, tmp_path, monkeypatch):
    """Both cases of the shape share the table; the conjugate one's temperature
    sweeps have no factored coefficients, which the two-ended form needs."""
    n = (48, 40, 6)
    two_ended(tmp_path / "tune.txt", n, [(1, 1, 0)])
    monkeypatch.setenv("LESGPU_AUTOTUNE", "1")
    monkeypatch.setenv("LESGPU_TUNE_FILE", str(tmp_path / "tune.txt"))
    plain = cases.cylinder(*n)
    a = leswht_gb300.gpu_solver(plain)
    a.step()
    assert (1, 1, 0, 272) in leswht_gb300.tuning(a.lib, a.h)
    case = cases.with_conjugate(plain, 2.0, 5.0)
    b, r = leswht_gb300.gpu_solver(case), solver.Solver(oracle_lib, "ref_", case)
    b.step(); r.step()
    assert other(b) == 0
    fb, fr = b.fields(), r.fields()
    for k in ("u", "v", "w", "p", "t"):
        assert np.linalg.norm(fb[k] - fr[k]) <= 1e-10 * max(np.linalg.norm(fr[k]), 1e-300), k
