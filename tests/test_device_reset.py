"""The library after its program reset the device (cudaDeviceReset ends the
program's own context): nothing kept of the old context is used
(tests/cpp/device_reset.cu, sharing the library's CUDA runtime)."""

import subprocess

import pytest

from tests import _native


@pytest.mark.gpu
def test_gpu_uses_before_and_after_a_reset(gpu):
    program = _native.build("device_reset.cu", "-cudart", "shared")
    result = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
