"""The two-ended FP64 sweeps (the tuned table's code 272) on every class of a
case, put there through the tuning file, against the oracle: periodic and
walled lines of even and odd lengths down to the shortest, batches that do not
fill a warp's 16 lines, in place (z), to scratch (y) and adding (x).  Bound:
the step's parity bound, 1e-10 of each field's norm."""
import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases, solver

pytestmark = pytest.mark.gpu

CASES = [
    ("channel", lambda: cases.channel(10, 9, 6), (1, 1)),
    ("channel", lambda: cases.channel(12, 5, 3), (1, 1)),
    ("channel", lambda: cases.channel(27, 32, 45), (1, 1)),
    ("channel", lambda: cases.channel(64, 65, 20), (1, 1)),
    ("channel", lambda: cases.channel(20, 130, 12), (1, 1)),
    ("duct", lambda: cases.with_poisson(cases.channel(36, 28, 20, zwalls=True), abi.POISSON_X_FT, nlev=1), (1, 0)),
    ("body", lambda: cases.cylinder(44, 36, 6), (0, 1)),
]


@pytest.mark.parametrize("q", range(len(CASES)))
def test_every_class_two_ended(oracle_lib, tmp_path, monkeypatch, q):
    _, build, (xper, zper) = CASES[q]
    case = build()
    n = (case.grid.n1m, case.grid.n2m, case.grid.n3m)
    path = tmp_path / "tune.txt"
    path.write_text("".join(f"adi {n[0]} {n[1]} {n[2]} {d} {nc} 0 {per} {ln} 272\n"
                            for d, per, ln in ((0, xper, n[0]), (1, 0, n[1]), (2, zper, n[2])) for nc in (1, 3)))
    monkeypatch.setenv("LESGPU_AUTOTUNE", "1")
    monkeypatch.setenv("LESGPU_TUNE_FILE", str(path))
    g, r = leswht_gb300.gpu_solver(case), solver.Solver(oracle_lib, "ref_", case)
    assert [w for d, nc, f32, w in leswht_gb300.tuning(g.lib, g.h) if d < 3] == [272] * 6
    for _ in range(2):
        g.step(); r.step()
    fg, fr = g.fields(), r.fields()
    for k in ("u", "v", "w", "p", "t"):
        assert np.linalg.norm(fg[k] - fr[k]) <= 1e-10 * max(np.linalg.norm(fr[k]), 1e-300), k
