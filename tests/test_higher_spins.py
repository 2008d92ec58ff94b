"""Spins above 2 (the spherical-harmonic tables' closed form at the lowest
degree, WignerStart in csrc/sht.cu): every basis function of a small grid
against Wigner's explicit sum, which is exact to a few 1e-15 of its terms at
these degrees; the recurrence adds a rounding or two a degree. 1e-13 covers
both."""

import math

import numpy as np
import pytest


def _wigner(l, m, N, theta):
    """d^l_{m N}(theta), Wigner's sum."""
    f = math.factorial
    c, s = np.cos(theta / 2), np.sin(theta / 2)
    total = np.zeros_like(theta)
    for k in range(max(0, N - m), min(l + N, l - m) + 1):
        total += (-1) ** (m - N + k) * c ** (2 * l + N - m - 2 * k) * s ** (m - N + 2 * k) / (
            f(l + N - k) * f(k) * f(m - N + k) * f(l - m - k))
    return math.sqrt(f(l + m) * f(l - m) * f(l + N) * f(l - N)) * total


@pytest.mark.gpu
@pytest.mark.parametrize("N", [-7, -4, -3, -2, -1, 0, 1, 2, 3, 5])
def test_gpu_basis_functions(gpu, N):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax = 8
    grid = SurfaceGrid(lmax, 7, 1.0)
    count = grid.SpinCoefficientSize(N)
    fields = grid.SynthesiseSpinBatch(N, torch.eye(count, dtype=torch.complex128, device=gpu).view(-1), count)
    fields = fields.view(count, grid.ntheta, grid.nphi)[:, :, 0].cpu().numpy()  # the meridian phi = 0
    for l in range(abs(N), lmax + 1):
        for m in range(-l, l + 1):
            want = math.sqrt((2 * l + 1) / (4 * math.pi)) * _wigner(l, m, N, grid.theta)
            got = fields[grid.SpinIndex(N, l, m)]
            assert np.max(np.abs(got - want)) < 1e-13, (l, m)


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 12])
def test_gpu_spin_1000(gpu, count):
    """A spin as large as a grid of degree 1000 has, whose only degree is its
    lowest. Its basis functions are orthogonal under the quadrature; each value
    is a product of up to 2000 roundings, so a round trip is within 1e-11."""
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax = N = 1000
    grid = SurfaceGrid(lmax, N, 1.0)
    c = torch.randn(count * grid.SpinCoefficientSize(N), dtype=torch.complex128, device=gpu,
                    generator=torch.Generator(device=gpu).manual_seed(N))
    back = grid.ExpandSpinBatch(N, grid.SynthesiseSpinBatch(N, c, count), count)
    assert float((back - c).abs().max()) < 1e-11 * float(c.abs().max())
