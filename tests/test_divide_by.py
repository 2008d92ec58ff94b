"""Division by stored reciprocals, as the strain's kernels divide, against
division (tests/cpp/divide_by.cu, on the host: the arithmetic is the device's)."""

import subprocess

from tests import _native


def test_divide_by_is_division():
    result = subprocess.run([str(_native.build("divide_by.cu"))], capture_output=True, text=True, timeout=300)
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
