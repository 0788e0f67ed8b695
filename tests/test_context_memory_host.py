"""Device memory of a context (csrc/context.hpp): blocks that a closed session
leaves for the next one never stand in the way of other calls and stay within
the context's cap.  tests/native/context_memory_check.cpp runs the allocation
code on the host against an accounted device of 300 MB."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_kept_blocks_give_way(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("g++ or CUDA's headers are not available")
    exe = str(tmp_path / "context_memory_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"), "-o", exe,
                    os.path.join(HERE, "native", "context_memory_check.cpp")], check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
