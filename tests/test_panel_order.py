"""A grid's table panels (the Legendre tables split for the tensor cores,
csrc/sht.cu) are made by the first call that wants one, on its stream. Calls on
other streams wait for them: the waits are asserted on the source, the results
of two streams' first calls against each other, and a capture right after the
first call against the call itself, bit for bit."""

import ctypes
import pathlib

import pytest

SHT = pathlib.Path(__file__).resolve().parent.parent / "sl3dpp_gb300" / "csrc" / "sht.cu"


@pytest.mark.parametrize("panels,launch,contract", [("panels64_", "LaunchPanelA64(", "Contract64("),
                                                     ("panels_", "LaunchPanelA(", "RunGemmTc(")])
def test_every_call_waits_for_the_panels(panels, launch, contract):
    text = SHT.read_text()
    wait = "if (int st = AwaitPanels(stream); st != SL3DGPU_OK) return st;"
    find = text.index(f"auto found = {panels}.find(key);")
    assert text[:find].rstrip().endswith(wait)
    body = text[find:]
    body = body[:body.index("\n}\n")]
    order = [body.index(t) for t in (launch, "MakePanel(stream, launch)", f"{panels}.emplace(", contract)]
    assert order == sorted(order)
    made = text[text.index("int Grid::MakePanel("):]
    made = made[:made.index("\n}\n")]
    assert made.index("launch(stream)") < made.index("cudaEventRecord(panelsMade_, stream)") < made.index(
        "panelsPending_ = true;")


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


@pytest.mark.gpu
@pytest.mark.parametrize("emulation", [False, True])
def test_gpu_capture_after_the_first_call(gpu, emulation):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid

    lmax, N, count = 48, -1, 12
    grid = SurfaceGrid(lmax, 2, 1.5, fp64_emulation=emulation)
    rng = torch.Generator(device=gpu).manual_seed(1)
    c = torch.randn(count * grid.SpinCoefficientSize(N), dtype=torch.complex128, device=gpu, generator=rng)
    later = torch.randn(c.shape, dtype=torch.complex128, device=gpu, generator=rng)
    grid.ExpandSpinBatch(N, grid.SynthesiseSpinBatch(N, c, count), count)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fields = grid.SynthesiseSpinBatch(N, c, count)
        back = grid.ExpandSpinBatch(N, fields, count)
    for values in (c.clone(), later):
        c.copy_(values)
        graph.replay()
        torch.cuda.synchronize()
        want = grid.SynthesiseSpinBatch(N, values, count)
        assert torch.equal(fields, want)
        assert torch.equal(back, grid.ExpandSpinBatch(N, want, count))
