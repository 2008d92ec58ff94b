"""The sea-level workspace kept with a grid after a solve that failed for want
of memory (tests/cpp/failed_allocations.cu, run without a device)."""

import os
import subprocess

from tests import _native


def test_kept_workspace_after_a_failed_allocation():
    result = subprocess.run([str(_native.build("failed_allocations.cu"))], capture_output=True, text=True, timeout=120,
                            env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    print(result.stdout)
    assert result.returncode == 0, result.stdout + result.stderr
