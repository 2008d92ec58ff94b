"""One grid called from several host threads, each on its own stream: the
Legendre stage, whose tables, batches and panels the grid makes on first use,
and whole sea-level solves. Every thread's results are the single thread's,
bit for bit."""

import ctypes
import threading

import numpy as np
import pytest


def _in_threads(work, count):
    failed = []

    def run(i):
        try:
            work(i)
        except BaseException as e:  # noqa: BLE001 -- reported below
            failed.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.gpu
def test_gpu_legendre_from_several_threads(gpu):
    import torch

    from sl3dpp_gb300._lib import check, lib
    from sl3dpp_gb300.grid import SurfaceGrid

    lmax = 40
    f = lib().sl3dgpu_legendre_device
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p] + [ctypes.c_int] * 4 + [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                                                           ctypes.c_void_p]
    grid, alone = SurfaceGrid(lmax, 2, 1.5), SurfaceGrid(lmax, 2, 1.5)
    calls = []
    for i, (N, count) in enumerate([(-2, 12), (-1, 12), (0, 12), (-2, 20), (1, 3), (-1, 30)]):
        x = torch.randn(grid.SpinCoefficientSize(N), count, dtype=torch.complex128, device=gpu,
                        generator=torch.Generator(device=gpu).manual_seed(i))
        shape = ((2 * lmax + 1) * grid.ntheta, count)
        calls.append((N, count, x, torch.zeros(shape, dtype=torch.complex128, device=gpu),
                      torch.zeros(shape, dtype=torch.complex128, device=gpu), torch.cuda.Stream()))
    for N, count, x, want, _, _ in calls:
        check(f(alone._handle, N, 0, 0, 0, x.data_ptr(), count, want.data_ptr(), None))
    torch.cuda.synchronize()

    def work(i):
        N, count, x, _, got, stream = calls[i]
        check(f(grid._handle, N, 0, 0, 0, x.data_ptr(), count, got.data_ptr(), stream.cuda_stream))

    _in_threads(work, len(calls))
    torch.cuda.synchronize()
    for N, count, _, want, got, _ in calls:
        assert torch.equal(got, want), (N, count)


@pytest.mark.gpu
def test_gpu_sea_level_solves_from_several_threads(gpu):
    import torch

    from sl3dpp_gb300.grid import SurfaceGrid
    from sl3dpp_gb300.sealevel import SeaLevelSolver
    from tests.test_sealevel import problem

    lmax = 24
    p = problem(lmax)
    solver = SeaLevelSolver(SurfaceGrid(lmax, 0, 1.0), p["h"], p["k"], p["lt"], None, None, None, 1.0, 1.0, 1.0)
    ocean = torch.tensor(p["ocean"], device=gpu)
    loads = [torch.tensor(p["load"] * (i + 1), device=gpu) for i in range(4)]
    torch.cuda.synchronize()
    solve = lambda i: solver.solve_generalised(ocean, rtol=1e-10, direct_load=loads[i])["sea_level_change"].cpu().numpy()
    want = [solve(i) for i in range(len(loads))]
    got = [None] * len(loads)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                got[i] = solve(i)

    _in_threads(work, len(loads))
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
