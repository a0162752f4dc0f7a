"""CPU: what a handle does when device memory cannot be had, over a fake of the allocation calls
(tests/device_memory_check.cpp against dm-heom_b200/csrc/device_memory.hpp)."""
import os
import subprocess

import pytest

CUDA = "/usr/local/cuda/include"


def test_failed_allocations_leave_no_half_made_state(tmp_path, root):
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    exe = tmp_path / "device_memory_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CUDA, "-I", os.path.join(root, "include"),
                    "-I", os.path.join(root, "dm-heom_b200", "csrc"), "-o", str(exe),
                    os.path.join(root, "tests", "device_memory_check.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout[-2000:]
