"""lesgpu_poisson_ftft_noalloc against the same solve in numpy -- FFT in x and
z, the y systems by a dense solve, the mean mode pinned -- over every radix
and mix of them, odd and even row counts down to two (the elimination meets in
the middle) and numbers of modes that leave half-warps part empty.  Bound: the
lowest wavenumbers' systems have condition numbers up to 1e5, so 1e-11 of
phi's norm."""
import ctypes as C

import numpy as np
import pytest

import leswht_gb300
from leswht_gb300 import abi, cases

pytestmark = pytest.mark.gpu

SIZES = [(4, 2, 2), (3, 3, 5), (5, 4, 3), (8, 5, 9), (6, 17, 25), (16, 16, 15), (30, 33, 24), (27, 64, 20), (125, 7, 8),
         (64, 81, 60), (128, 10, 128)]


def reference(g, div):
    n1, n2, n3 = g.n1m, g.n2m, g.n3m
    rhs = np.fft.fft2(div, axes=(0, 2))
    kx = 2.0 * (1.0 - np.cos(2.0 * np.pi * np.arange(n1) / n1)) * g.f2fxi[1] ** 2
    kz = 2.0 * (1.0 - np.cos(2.0 * np.pi * np.arange(n3) / n3)) * g.f2fzi[1] ** 2
    lo = np.array([0.0] + [g.f2fyi[j] * g.c2cyi[j] for j in range(2, n2 + 1)])
    up = np.array([g.f2fyi[j] * g.c2cyi[j + 1] for j in range(1, n2)] + [0.0])
    A = np.diag(-(lo + up)) + np.diag(lo[1:], -1) + np.diag(up[:-1], 1)
    M = A[None, None] - (kz[:, None] + kx[None, :])[:, :, None, None] * np.eye(n2)
    b = rhs.transpose(0, 2, 1).copy()
    ref = b[0, 0, -1]
    M[0, 0, -1] = 0.0
    M[0, 0, -1, -1] = 1.0
    b[0, 0, -1] = 0.0
    x = np.linalg.solve(M, b[..., None])[..., 0]
    x[0, 0] -= (ref - lo[-1] * x[0, 0, -2]) / -(lo[-1] + up[-1])
    x[0, 0, -1] = 0.0
    return np.fft.ifft2(x.transpose(0, 2, 1), axes=(0, 2)).real


@pytest.mark.parametrize("n1,n2,n3", SIZES)
def test_matches_numpy(n1, n2, n3):
    torch = pytest.importorskip("torch")
    fn = leswht_gb300.load_library().lesgpu_poisson_ftft_noalloc
    fn.argtypes = [C.POINTER(abi.Grid), C.c_void_p, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    g = cases.channel(n1, n2, n3).grid
    d = np.random.default_rng(5).standard_normal((n3, n2, n1))
    wy = g.f2fy[None, 1:n2 + 1, None]
    d -= (d * wy).sum() / (wy.sum() * n1 * n3)
    full = np.zeros(g.shape)
    full[1:n3 + 1, 1:n2 + 1, 1:n1 + 1] = d
    dd = torch.from_numpy(full).cuda()
    phi = torch.full(g.shape, np.nan, dtype=torch.float64, device="cuda")
    assert fn(C.byref(abi.pack_grid(g).struct), dd.data_ptr(), phi.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    got, want = phi.cpu().numpy()[1:n3 + 1, 1:n2 + 1, 1:n1 + 1], reference(g, d)
    assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
