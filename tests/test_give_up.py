"""A bounded wait of the tensor-core contractions that gave up is reported by
the grid's next call (tests/cpp/give_up.cu, built against the library)."""

import subprocess

import pytest

from tests import _native


@pytest.mark.gpu
def test_gpu_a_wait_that_gave_up_is_reported(gpu):
    result = subprocess.run([str(_native.build("give_up.cu"))], capture_output=True, text=True, timeout=300)
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
