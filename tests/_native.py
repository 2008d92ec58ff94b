"""Test programs in CUDA C++ against the library's own headers (tests/cpp/*.cu),
compiled with the library's flags and linked to it."""

from __future__ import annotations

import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parent.parent


def build(source: str, *flags: str) -> pathlib.Path:
    """Compile tests/cpp/<source> and return the program's path."""
    import __graft_entry__
    from sl3dpp_gb300 import _lib
    from sl3dpp_gb300 import build as product

    __graft_entry__.build()
    path = ROOT / "tests" / "cpp" / source
    out = path.parent / "_build" / path.stem
    out.parent.mkdir(exist_ok=True)
    cmd = [product._nvcc(), *product.ARCH, *product.NVCC_FLAGS, *flags, str(path), "-o", str(out),
           "-L", str(_lib.LIBRARY_PATH.parent), "-lsl3dgpu", "-Xlinker", f"-rpath={_lib.LIBRARY_PATH.parent}"]
    result = subprocess.run(cmd, capture_output=True, text=True)
    assert result.returncode == 0, " ".join(cmd) + "\n" + result.stderr
    return out
