"""Rings of subnormal values, and rings under subnormal weights, in the FP64
longitude transforms: the fixed-point form holds neither, so both take the
FP64 units, as batches of few fields do (tests/cpp/ring_subnormals.cu, built
against the library, compares the two)."""

import subprocess

import pytest

from tests import _native


@pytest.mark.gpu
def test_gpu_rings_of_subnormals(gpu):
    result = subprocess.run([str(_native.build("ring_subnormals.cu"))], capture_output=True, text=True, timeout=300)
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
