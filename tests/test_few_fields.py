"""Calls of one to eight fields, whose Legendre sums read and write the
reference layout's coefficients themselves (LegendreInReferenceLayout,
csrc/sht.cu), against the same fields in a batch of nine, which goes through
the permutations and the other kernels.

Both are FP64 to a few 1e-15 of the largest value times the degrees' growth:
1e-13 of the largest."""

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,N,real", [(0, 0, True), (1, 0, True), (2, 0, True), (17, 0, True), (33, 0, True),
                                         (70, 0, True), (1, 1, False), (2, -2, False), (3, 2, False),
                                         (17, -1, False), (33, -2, False), (70, 0, False)])
def test_gpu_few_fields_follow_the_batch(gpu, lmax, N, real):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    grid = SurfaceGrid(lmax, min(2, lmax), 1.0)
    synthesise = grid.SynthesiseBatch if real else lambda c, n: grid.SynthesiseSpinBatch(N, c, n)
    expand = grid.ExpandBatch if real else lambda f, n: grid.ExpandSpinBatch(N, f, n)
    size = grid.CoefficientSize() if real else grid.SpinCoefficientSize(N)
    rng = torch.Generator(device=gpu).manual_seed(lmax)
    c = torch.randn(9, size, dtype=torch.complex128, device=gpu, generator=rng)
    f = torch.randn(9, grid.FieldSize(), dtype=torch.float64 if real else torch.complex128, device=gpu, generator=rng)
    fields = synthesise(c.reshape(-1), 9).view(9, -1)
    coefficients = expand(f.reshape(-1), 9).view(9, -1)
    for count in range(1, 9):
        few = synthesise(c[:count].reshape(-1), count).view(count, -1)
        assert float((few - fields[:count]).abs().max()) <= 1e-13 * float(fields.abs().max()), count
        few = expand(f[:count].reshape(-1), count).view(count, -1)
        assert float((few - coefficients[:count]).abs().max()) <= 1e-13 * float(coefficients.abs().max()), count
