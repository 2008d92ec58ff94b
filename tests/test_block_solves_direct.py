"""The Cholesky solves by blocks of rows, called directly at either block size,
in FP64 and over row windows in FP32: tests/cpp/block_solves.cu, built against
the library, states the bound that each solution's backward error is held to."""

import subprocess

import pytest

from tests import _native


@pytest.mark.gpu
def test_gpu_blocked_solves_directly(gpu):
    result = subprocess.run([str(_native.build("block_solves.cu"))], capture_output=True, text=True, timeout=300)
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
    assert "blocks of 8\n" in result.stdout and "blocks of 16\n" in result.stdout
