"""The default FP64 Legendre contraction on the tensor cores (eight BF16
slices) against the narrow kernels on the FP64 units, which a batch of one
field takes: the same column alone, at the tiles' edges (columns over 16 and
64, rows over 128, depths over 16) and, for columns with infinities or NaN,
the same pattern of non-finite results.

Tolerance: a value enters with an error below 2^-57 of its row's (column's)
largest and the dropped products stay below 7 2^-58 of the two maxima a
term, so a result of depth K is within K 2^-54 of (row maximum) x (column
maximum); the FP64 units' own sum is within K 2^-53 of it. Together below
K 2^-52, which the largest row and column maxima bound for every value."""

import ctypes

import numpy as np
import pytest


def _legendre(grid, N, real, analysis, x, count, out):
    from sl3dpp_gb300._lib import check, lib

    f = lib().sl3dgpu_legendre_device
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 4 + [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                                                           ctypes.c_void_p]
    check(f(grid._handle, N, int(real), int(analysis), 0, x.data_ptr(), count, out.data_ptr(), None))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,N,real,oversampling,count",
                         [(3, -2, False, 1.0, 9), (15, 0, True, 1.0, 32), (16, -1, False, 1.5, 33),
                          (63, 0, True, 1.0, 10), (85, -2, False, 1.5, 17), (128, -1, False, 1.0, 40),
                          (256, 0, True, 1.5, 9)])
def test_gpu_slices_match_the_fp64_units(gpu, lmax, N, real, oversampling, count):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    g = SurfaceGrid(lmax, 2, oversampling)
    rows = g.CoefficientSize() if real else g.SpinCoefficientSize(N)
    orders = lmax + 1 if real else 2 * lmax + 1
    torch.manual_seed(lmax + count)
    for analysis in (False, True):
        inner = orders * g.ntheta if analysis else rows
        outer = rows if analysis else orders * g.ntheta
        x = torch.randn(inner, count, dtype=torch.complex128, device=gpu)
        x[:, 1] *= 1e-200  # columns keep their own exponents
        x[:, 2] *= 1e150
        x[:, 3] = 0.0
        got = _legendre(g, N, real, analysis, x, count, torch.empty(outer, count, dtype=torch.complex128, device=gpu))
        depth = g.ntheta if analysis else lmax + 1
        table = np.sqrt((2 * lmax + 1) / (4 * np.pi))  # |d| <= 1
        for p in (0, 1, 2, 3, count - 1):
            alone = _legendre(g, N, real, analysis, x[:, p].contiguous(), 1,
                              torch.empty(outer, 1, dtype=torch.complex128, device=gpu))
            largest = float(torch.view_as_real(x[:, p]).abs().max())
            error = float(torch.view_as_real(got[:, p] - alone[:, 0]).abs().max())
            assert error <= depth * 2.0**-52 * table * largest, (analysis, p)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_gpu_slices_keep_non_finite_columns(gpu, bad):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax, count = 20, 20
    g = SurfaceGrid(lmax, 2, 1.5)
    orders, rows = 2 * lmax + 1, g.SpinCoefficientSize(-1)
    torch.manual_seed(1)
    for analysis in (False, True):
        inner, outer = (orders * g.ntheta, rows) if analysis else (rows, orders * g.ntheta)
        x = torch.randn(inner, count, dtype=torch.complex128, device=gpu)
        x[inner // 2, 4] = complex(bad, 1.0)
        x[inner // 3, 17] = complex(0.0, -bad)
        got = _legendre(g, -1, False, analysis, x, count, torch.empty(outer, count, dtype=torch.complex128, device=gpu))
        for p in range(count):
            alone = _legendre(g, -1, False, analysis, x[:, p].contiguous(), 1,
                              torch.empty(outer, 1, dtype=torch.complex128, device=gpu))[:, 0]
            a, b = torch.view_as_real(got[:, p]), torch.view_as_real(alone)
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
            assert torch.equal(a[torch.isinf(a)], b[torch.isinf(b)])
            assert bool(torch.isfinite(a).all()) == (p not in (4, 17))
