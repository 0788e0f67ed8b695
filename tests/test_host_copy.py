"""The staged copies between pageable memory and the device (csrc/host_copy.cu),
run on the host by tests/native/host_copy_check.cpp: CUDA's calls are replaced
by streams whose copies stay in flight until they are asked about, the helper
threads are real.  Sizes around a slot and around each rule's limit, no memory
to pin, several threads and contexts, contexts that close while others open,
copies that fail on the way."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("g++ or CUDA's headers are not available")
    exe = str(tmp_path_factory.mktemp("host_copy") / "host_copy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"), "-o", exe,
                    os.path.join(HERE, "native", "host_copy_check.cpp"), "-lpthread"], check=True,
                   capture_output=True)
    return exe


@pytest.mark.parametrize("check", ["sizes", "ways", "pins", "pinned_by_the_caller", "no_slots", "threads", "helpers_live", "failing_copy"])
def test_copies(program, check):
    out = subprocess.run([program, check], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
