"""Host harnesses of the library's native code: ``tests/native/*.cu`` compiled with the
library's own flags, for tests that call them through ctypes without a GPU."""

import ctypes
import os
import subprocess

import pytest

from pycfd_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(name, out_dir):
    """Compile ``tests/native/<name>.cu`` into ``out_dir`` and load it."""
    so = os.path.join(str(out_dir), f"lib{name}.so")
    cmd = [build.nvcc(), *build.NVCC_FLAGS, "-O1", "-Wno-deprecated-gpu-targets", "-o", so,
           os.path.join(HERE, "native", f"{name}.cu")]
    try:
        done = subprocess.run(cmd, capture_output=True, text=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")
    assert done.returncode == 0, done.stderr[-3000:]
    return ctypes.CDLL(so)
