"""lesgpu_poisson_ftft_noalloc on sizes that fill its fixed scratch to within
600 bytes of the limit (the tables of the y rows take a few kilobytes of it),
and on ones a step beyond, which it refuses.  phi against FFT and elimination
in numpy; the lowest wavenumbers' systems of some hundred rows have condition
numbers up to 1e6, so 1e-10 of phi's norm."""
import ctypes as C

import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def solve(g, div):
    n1, n2, n3 = g.n1m, g.n2m, g.n3m
    b = np.fft.fft(np.fft.rfft(div, axis=0), axis=2).transpose(1, 0, 2).copy()
    kx = 2.0 * (1.0 - np.cos(2.0 * np.pi * np.arange(n1) / n1)) * g.f2fxi[1] ** 2
    kz = 2.0 * (1.0 - np.cos(2.0 * np.pi * np.arange(n3 // 2 + 1) / n3)) * g.f2fzi[1] ** 2
    k2 = kz[:, None] + kx[None, :]
    lo = np.array([0.0] + [g.f2fyi[j] * g.c2cyi[j] for j in range(2, n2 + 1)])
    up = np.array([g.f2fyi[j] * g.c2cyi[j + 1] for j in range(1, n2)] + [0.0])
    ref = b[-1, 0, 0]
    gam = np.zeros_like(b, dtype=np.float64)
    for j in range(n2):
        d, l = -(lo[j] + up[j] + k2), np.full_like(k2, lo[j])
        if j == n2 - 1:
            d[0, 0], l[0, 0], b[j, 0, 0] = 1.0, 0.0, 0.0
        if j:
            d = d - l * gam[j - 1]
            b[j] = b[j] - l * b[j - 1]
        b[j] /= d
        gam[j] = up[j] / d
    for j in range(n2 - 2, -1, -1):
        b[j] -= gam[j] * b[j + 1]
    b[:-1, 0, 0] -= (ref - lo[-1] * b[-2, 0, 0]) / -(lo[-1] + up[-1])
    return np.fft.irfft(np.fft.ifft(b.transpose(1, 0, 2), axis=2), n=n3, axis=0)


def call(g, dd, phi):
    torch = pytest.importorskip("torch")
    fn = leswht_gb300.load_library().lesgpu_poisson_ftft_noalloc
    fn.argtypes = [C.POINTER(abi.Grid), C.c_void_p, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    return fn(C.byref(abi.pack_grid(g).struct), dd.data_ptr(), phi.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("n1,n2,n3", [(18, 248, 625), (40, 217, 320), (12, 453, 512)])
def test_at_the_limit(n1, n2, n3):
    torch = pytest.importorskip("torch")
    g = cases.channel(n1, n2, n3).grid
    d = np.random.default_rng(5).standard_normal((n3, n2, n1))
    wy = g.f2fy[None, 1:n2 + 1, None]
    d -= (d * wy).sum() / (wy.sum() * n1 * n3)
    full = np.zeros(g.shape)
    full[1:n3 + 1, 1:n2 + 1, 1:n1 + 1] = d
    phi = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    assert call(g, torch.from_numpy(full).cuda(), phi) == 0
    got, want = phi.cpu().numpy()[1:n3 + 1, 1:n2 + 1, 1:n1 + 1], solve(g, d)
    assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("n1,n2,n3", [(18, 249, 625), (40, 218, 320), (12, 454, 512)])
def test_beyond_it(n1, n2, n3):
    torch = pytest.importorskip("torch")
    g = cases.channel(n1, n2, n3).grid
    phi = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    assert call(g, torch.zeros_like(phi), phi) == abi.ERR_TOO_LARGE
