"""The branch-free pivot reciprocal of the two-ended sweeps.  Its seed is off
by less than 2^-22, the third-order step leaves the cube of that, 2^-66, and
the last multiply-add rounds: 2 ulp with room.  It declares itself valid where
operand and result are normal with a margin, exponents of -923 to 923, and not
for zeros, denormals, infinities and NaN, which the sweep then divides."""
import ctypes as C

import numpy as np
import pytest

import leswht_gb300

pytestmark = pytest.mark.gpu


def reciprocal(x):
    fn = leswht_gb300.load_library().lesgpu_check_rcp_fast
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64]
    fn.restype = C.c_int
    x = np.ascontiguousarray(np.concatenate([x, -np.asarray(x)]), dtype=np.float64)
    r, ok = np.empty_like(x), np.empty_like(x)
    assert fn(x.ctypes.data, r.ctypes.data, ok.ctypes.data, x.size) == 0
    return x, r, ok == 1.0


def test_within_two_ulp():
    rng = np.random.default_rng(6)
    x = np.ldexp(rng.uniform(1.0, 2.0, 200000), rng.integers(-923, 924, 200000))
    low, high = 2.0 ** -923, np.nextafter(2.0 ** 924, 0.0)
    x = np.concatenate([x, rng.uniform(0.5, 2.0, 100000), [1.0, 3.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), low,
                        np.nextafter(low, 1.0), high, 2.0 ** 923]])
    x, r, ok = reciprocal(x)
    assert ok.all()
    exact = 1.0 / x
    assert np.all(np.abs(r - exact) <= 2.0 * np.spacing(np.abs(exact)))


def test_declines():
    x = [0.0, np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** 1023, np.nextafter(2.0 ** -923, 0.0), 2.0 ** 924]
    assert not reciprocal(x)[2].any()
