"""A grid's table panels (the Legendre tables split for the tensor cores,
csrc/sht.cu) are made by the first call that wants one, on that call's stream.
A call on another stream finds the panel made, so it must be finished by
then: the waits are asserted on the source, and the second stream's results
against the first's, whose stream made the panel, bit for bit."""

import ctypes
import pathlib

import pytest

SHT = pathlib.Path(__file__).resolve().parent.parent / "sl3dpp_gb300" / "csrc" / "sht.cu"


@pytest.mark.parametrize("panels", ["panels64_", "panels_"])
def test_a_panel_is_finished_before_another_call_can_find_it(panels):
    """The wait comes after the call's launches, whatever their status, and
    before the call returns (C calls hold the grid's lock until then)."""
    text = SHT.read_text()
    made = text.index(f"found = {panels}.emplace(")
    rest = text[made:text.index("\n}\n", made)]
    after = rest[rest.index("const int status ="):]
    assert "if (made) SL3D_CUDA(cudaStreamSynchronize(stream));" in after
    assert "return" not in after[:after.index("if (made)")]


@pytest.mark.gpu
@pytest.mark.parametrize("analysis", [False, True])
@pytest.mark.parametrize("fp32,emulation", [(False, False), (False, True), (True, False)])
def test_gpu_first_calls_on_two_streams(gpu, analysis, fp32, emulation):
    import torch

    from sl3dpp_gb300._lib import check, lib
    from sl3dpp_gb300.grid import SurfaceGrid

    lmax, N, count = 96, -2, 24
    f = lib().sl3dgpu_legendre_device
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 4 + [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                                                           ctypes.c_void_p]
    grid = SurfaceGrid(lmax, 2, 1.5, fp64_emulation=emulation)
    rows, rings = grid.SpinCoefficientSize(N), (2 * lmax + 1) * grid.ntheta
    kind = torch.complex64 if fp32 else torch.complex128
    x = torch.randn(rings if analysis else rows, count, dtype=kind, device=gpu,
                    generator=torch.Generator(device=gpu).manual_seed(lmax))
    outs = [torch.zeros(rows if analysis else rings, count, dtype=kind, device=gpu) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for stream, out in zip(streams, outs):
        check(f(grid._handle, N, 0, int(analysis), int(fp32), x.data_ptr(), count, out.data_ptr(), stream.cuda_stream))
    torch.cuda.synchronize()
    assert float(outs[0].abs().max()) > 0.0
    assert torch.equal(outs[0], outs[1])
