"""The library's grow-only device buffer after a failed allocation, compiled for the
host (g++) with an allocator of its own."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_failed_growth_leaves_an_empty_buffer(tmp_path):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    exe = str(tmp_path / "device_buffer")
    src = os.path.join(ROOT, "tests", "cpp", "device_buffer.cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CUDA, "-o", exe, src], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
