"""The permutations between the reference's coefficients and the device rows
(PermuteKernel, csrc/sht.cu: tiles of 32 coefficients by 32 fields) around the
edges of a tile: batches whose field and coefficient counts leave a tile
short, full and just passed, against the same fields alone, which have no
permutation. Both sides are FP64 transforms: 1e-13 of the largest value."""

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,N,real", [(2, 0, True), (6, 0, True), (7, -1, False), (21, -2, False), (40, 0, True)])
@pytest.mark.parametrize("count", [9, 31, 32, 33, 65])
def test_gpu_permuted_batches_follow_single_fields(gpu, lmax, N, real, count):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    grid = SurfaceGrid(lmax, 2, 1.0)
    synthesise = grid.SynthesiseBatch if real else lambda c, n: grid.SynthesiseSpinBatch(N, c, n)
    expand = grid.ExpandBatch if real else lambda f, n: grid.ExpandSpinBatch(N, f, n)
    size = grid.CoefficientSize() if real else grid.SpinCoefficientSize(N)
    rng = torch.Generator(device=gpu).manual_seed(lmax + count)
    c = torch.randn(count, size, dtype=torch.complex128, device=gpu, generator=rng)
    f = torch.randn(count, grid.FieldSize(), dtype=torch.float64 if real else torch.complex128, device=gpu,
                    generator=rng)
    fields = synthesise(c.reshape(-1), count).view(count, -1)
    coefficients = expand(f.reshape(-1), count).view(count, -1)
    for p in range(0, count, 7):
        assert float((synthesise(c[p].contiguous(), 1) - fields[p]).abs().max()) <= 1e-13 * float(fields.abs().max())
        assert float((expand(f[p].contiguous(), 1) - coefficients[p]).abs().max()) <= 1e-13 * float(
            coefficients.abs().max())
