"""The FP64 Cholesky solves by blocks of rows (csrc/band_block.cu), at both
block sizes and with row counts that are and are not multiples of them: under
the conjugate-gradient step without lateral viscosity the preconditioner is
the operator, so the solve must end at once with K x = f. A first
iteration's residual is the solve's own error, far below 1e-10 of f."""

import numpy as np
import pytest

from sl3dpp_gb300 import configs


@pytest.mark.gpu
@pytest.mark.parametrize("lmax,elements,ngll,kelvin", [(2, 20, 5, 0.0), (9, 21, 6, 0.5), (16, 23, 5, 0.0),
                                                       (33, 40, 6, 0.0), (45, 43, 5, 0.5), (100, 70, 6, 0.0)])
def test_gpu_blocked_solves_invert_the_systems(gpu, lmax, elements, ngll, kelvin):
    import torch

    from sl3dpp_gb300.viscoelastic3d import Options, Viscoelastic3D, standard_earth

    op = Viscoelastic3D(standard_earth(elements, kelvin, 10.0),
                        Options.defaults(lmax, ngll, solver=1, solve_rtol=1e-10, solve_max_iterations=4))
    op.set_delta(np.zeros(op.values))
    dt = 500 * configs.SECONDS_PER_YEAR / op.time_scale
    state = op.ZeroState()
    rng = np.random.default_rng(lmax)
    load = rng.standard_normal((lmax + 1) * (lmax + 2) // 2) + 0j
    step = op.StartStep(state, dt, "backward_euler", load)
    forces = step.Forces(load)
    # every row of every column, not only the load's
    noise = torch.randn(forces.numel(), dtype=torch.complex128, device=gpu,
                        generator=torch.Generator(device=gpu).manual_seed(lmax))
    wanted = step.Apply(noise * float(forces.abs().max()))
    x, info = step.Solve(wanted)
    assert info.solve_iterations <= 2, info.solve_iterations
    back = step.Apply(x)
    assert float((back - wanted).abs().max()) < 1e-9 * float(wanted.abs().max())
