"""The stage weights made once a block (csrc/step_kernels.cu: SpectralStart,
SpectralAdvance and Weights kernels), from a few nodes to about as many as
the force kernel takes: a model without lateral viscosity steps its memory
spectrally; with a pattern of 4e-16 everywhere it steps on the grid, through
the other kernels, under the same weights to rounding. The two must agree. A
wrong weight is an error of order one; rounding, amplified by the systems'
condition with thousands of nodes, stays far below 1e-6."""

import numpy as np
import pytest

from sl3dpp_gb300 import configs


@pytest.mark.gpu
@pytest.mark.parametrize("elements", [40, 500, 1000])
@pytest.mark.parametrize("scheme", [0, 1])
def test_gpu_spectral_and_grid_memories_agree(gpu, elements, scheme):
    from sl3dpp_gb300.viscoelastic3d import Options, Viscoelastic3D, standard_earth

    lmax = 2
    load = np.arange(1.0, 7.0) * 1e-4 + 0j
    found = []
    for lateral in (False, True):
        op = Viscoelastic3D(standard_earth(elements, 0.5, 10.0), Options.defaults(lmax, 6))
        if lateral:
            op.set_delta(np.full(op.values, 4e-16))
        state = op.ZeroState()
        dt = 500 * configs.SECONDS_PER_YEAR / op.time_scale
        for n in range(2):
            op.Step(state, dt, scheme, load * n, load * (n + 1))
        found.append(state.strain_coefficients())
    spectral, grid = found
    assert np.max(np.abs(spectral)) > 0.0
    assert np.max(np.abs(spectral - grid)) < 1e-6 * np.max(np.abs(spectral))
