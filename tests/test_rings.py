"""The longitude transforms of FP64 values in block fixed point
(csrc/ring_fixed.cu) at the sizes where they can go wrong: ring lengths from
1 through every radix of the plans, nine to seventeen fields (the CTA's groups,
the odd field of a real pair; batches of up to eight take the FP64 units),
values near the ends of the FP64 range and
non-finite ones, whose rings run in FP64.

Round trips are held to the transforms' bar, 1e-12 of the largest
coefficient; a power-of-two factor on the inputs must come through exactly."""

import numpy as np
import pytest


def _coefficients(torch, grid, N, real, count, device, seed):
    g = torch.Generator(device=device).manual_seed(seed)
    n = grid.CoefficientSize() if real else grid.SpinCoefficientSize(N)
    c = torch.randn(count, n, dtype=torch.complex128, device=device, generator=g)
    if real:
        zonal = torch.tensor([l * (l + 1) // 2 for l in range(grid.lmax + 1)], device=device)
        c[:, zonal] = c[:, zonal].real.to(torch.complex128)
    return c


def _round_trip(grid, N, real, c, count):
    if real:
        f = grid.SynthesiseBatch(c.reshape(-1).contiguous(), count)
        return f, grid.ExpandBatch(f, count).view(count, -1)
    f = grid.SynthesiseSpinBatch(N, c.reshape(-1).contiguous(), count)
    return f, grid.ExpandSpinBatch(N, f, count).view(count, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,oversampling", [(0, 1.0), (1, 1.0), (2, 1.0), (4, 1.0), (5, 1.0), (7, 1.0), (8, 1.5),
                                               (13, 1.0), (24, 1.0), (33, 1.5), (40, 1.0), (45, 1.5), (63, 1.0),
                                               (80, 1.0), (134, 1.0), (191, 1.0)])
def test_gpu_rings_round_trip(gpu, lmax, oversampling):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    grid = SurfaceGrid(lmax, min(2, lmax), oversampling)
    for N, real in ((0, True), (-min(2, lmax), False)):
        for count in (8, 9, 10, 17) if lmax < 100 else (9, 16):
            c = _coefficients(torch, grid, N, real, count, gpu, lmax + count)
            f, back = _round_trip(grid, N, real, c, count)
            assert float((back - c).abs().max()) < 1e-12 * float(c.abs().max()), (N, count)
            # the same field alone, on the FP64 units, under an exact factor
            one, _ = _round_trip(grid, N, real, c[count - 1:] * 2.0**-40, 1)
            last = f.view(count, -1)[count - 1]
            assert float((one * 2.0**40 - last).abs().max()) < 1e-13 * float(last.abs().max()), (N, count)


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [-960, 960])
def test_gpu_rings_near_the_ends_of_the_range(gpu, exponent):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    grid = SurfaceGrid(12, 2, 1.5)
    count = 10
    c = _coefficients(torch, grid, -1, False, count, gpu, 3)
    want, _ = _round_trip(grid, -1, False, c, count)
    c[1] *= 2.0**exponent
    got, back = _round_trip(grid, -1, False, c, count)
    got, want = got.view(count, -1), want.view(count, -1)
    for p, scale in ((0, 0), (1, exponent), (2, 0), (9, 0)):
        error = (got[p] * 2.0**-scale - want[p]).abs().max()
        assert float(error) < 1e-13 * float(want[p].abs().max())
        assert float((back[p] - c[p]).abs().max()) < 1e-12 * float(c[p].abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_gpu_rings_keep_non_finite_fields_apart(gpu, bad):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax, count = 10, 11
    grid = SurfaceGrid(lmax, 2, 1.5)
    for N, real in ((0, True), (-2, False)):
        c = _coefficients(torch, grid, N, real, count, gpu, 9)
        want, _ = _round_trip(grid, N, real, c, count)
        c[2, 7] = complex(bad, 0.0)
        got, _ = _round_trip(grid, N, real, c, count)
        got, want = got.view(count, -1), want.view(count, -1)
        assert not bool(torch.isfinite(torch.view_as_real(got[2]) if not real else got[2]).all())
        # a real field shares its ring with its pair, 2 with 3
        for p in (0, 1, 4, 10) if real else (0, 1, 3, 4, 10):
            assert float((got[p] - want[p]).abs().max()) < 1e-13 * float(want[p].abs().max())
        # and a field whose one value is bad: its coefficients are, the others' are not
        f = (grid.SynthesiseBatch if real else lambda x, n: grid.SynthesiseSpinBatch(N, x, n))(
            _coefficients(torch, grid, N, real, count, gpu, 9).reshape(-1).contiguous(), count).view(count, -1)
        f[4, 3] = bad
        e = (grid.ExpandBatch if real else lambda x, n: grid.ExpandSpinBatch(N, x, n))(f.reshape(-1).contiguous(), count)
        finite = torch.isfinite(torch.view_as_real(e)).view(count, -1).all(dim=1)
        # (of a real pair, 4 with 5, both)
        assert [p for p in range(count) if not finite[p]] == ([4, 5] if real else [4])
