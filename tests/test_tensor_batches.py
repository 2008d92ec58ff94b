"""The three components of a tensor in one launch (Grid::LegendreSynthesis3
and its fellows, csrc/sht.cu) against the components one at a time. The
lateral operator is linear in its pattern, and a pattern on one element (5
nodes) is few enough fields to go through the FP64 units a component at a
time; the same pattern on two elements (10 nodes) goes through the joint
launches. So the two elements' operators add up to the joint one.

Both sides are FP64 to a few 1e-15 of the largest term, and the common part
K x is in each: 1e-12 of the largest value leaves two digits."""

import numpy as np
import pytest

from sl3dpp_gb300 import configs


@pytest.mark.gpu
@pytest.mark.parametrize("lmax", [2, 3, 9, 16, 33, 50])
def test_gpu_joint_components_add_up(gpu, lmax):
    import torch

    from sl3dpp_gb300.viscoelastic3d import Options, Viscoelastic3D, standard_earth

    op = Viscoelastic3D(standard_earth(20, 0.0, 10.0), Options.defaults(lmax, 5, solver=1))
    dt = 500 * configs.SECONDS_PER_YEAR / op.time_scale
    nodes = op.node_count
    rng = np.random.default_rng(lmax)
    pattern = 0.5 * rng.standard_normal((nodes, op.values // nodes))
    load = rng.standard_normal((lmax + 1) * (lmax + 2) // 2) + 0j
    noise = None
    applied = []
    first = nodes // 10 * 5  # an element of the mantle
    for lo, hi in ((0, 0), (first, first + 5), (first + 5, first + 10), (first, first + 10)):
        delta = np.zeros_like(pattern)
        delta[lo:hi] = pattern[lo:hi]
        op.set_delta(delta.ravel())
        step = op.StartStep(op.ZeroState(), dt, "backward_euler", load)
        if noise is None:
            noise = torch.randn(step.Forces(load).numel(), dtype=torch.complex128, device=gpu,
                                generator=torch.Generator(device=gpu).manual_seed(lmax))
        applied.append(step.Apply(noise))
        step.Finish()
    none, a, b, both = applied
    scale = float(none.abs().max())
    assert float((both - none).abs().max()) > 1e-8 * scale  # the pattern is felt
    assert float((a + b - none - both).abs().max()) < 1e-12 * scale
