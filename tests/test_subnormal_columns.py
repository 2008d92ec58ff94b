"""Columns of subnormal values in the default FP64 Legendre contraction (eight
BF16 slices, csrc/tc_gemm64.cu): subnormal values have one exponent whatever
their leading bit, so such a column is split by its own shift. Against the
same column alone, on the FP64 units.

Tolerance: both sums are over the exact values within the bound of
tests/test_slices.py (depth x 2^-52 of the two maxima), which for subnormal
columns is below the spacing 2^-1074 of the results; each result is rounded
to that spacing, the FP64 units' once a term. So depth + 1 spacings."""

import ctypes

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
def test_gpu_subnormal_columns(gpu):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax, N, count = 20, -1, 12
    grid = SurfaceGrid(lmax, 2, 1.5)
    rows, rings = grid.SpinCoefficientSize(N), (2 * lmax + 1) * grid.ntheta
    for analysis in (False, True):
        inner, outer = (rings, rows) if analysis else (rows, rings)
        x = torch.rand(inner, count, dtype=torch.complex128, device=gpu,
                       generator=torch.Generator(device=gpu).manual_seed(7))
        # the largest just normal, just subnormal, and far into the subnormals
        exponents = {1: -1021, 2: -1022, 3: -1023, 4: -1030, 5: -1060}
        for p, e in exponents.items():
            x[:, p] = x[:, p] * 2.0**-500 * 2.0 ** (e + 500)
        got = _legendre(grid, N, False, analysis, x, count, torch.empty(outer, count, dtype=torch.complex128, device=gpu))
        depth = grid.ntheta if analysis else lmax + 1
        for p in exponents:
            alone = _legendre(grid, N, False, analysis, x[:, p].contiguous(), 1,
                              torch.empty(outer, 1, dtype=torch.complex128, device=gpu))
            # brought into the normal range, exactly
            a, b = (torch.view_as_real(v) * 2.0**600 for v in (got[:, p], alone[:, 0]))
            assert float(b.abs().max()) > 0.0
            assert float((a - b).abs().max()) <= (depth + 1) * 2.0 ** (-1074 + 600), (analysis, p)
