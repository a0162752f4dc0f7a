"""CPU: what a handle does when device memory cannot be had, and the flags that handles share, over a fake of the
CUDA calls (tests/device_memory_check.cpp against dm-heom_b200/csrc/device_memory.hpp, tests/host_flag_check.cpp
against host_flag.hpp)."""
import os
import subprocess

import pytest

CUDA = "/usr/local/cuda/include"


def run_check(tmp_path, root, name):
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("CUDA headers not available")
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CUDA, "-I", os.path.join(root, "include"),
                    "-I", os.path.join(root, "dm-heom_b200", "csrc"), "-o", str(exe),
                    os.path.join(root, "tests", name + ".cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout[-2000:]


def test_failed_allocations_leave_no_half_made_state(tmp_path, root):
    run_check(tmp_path, root, "device_memory_check")


def test_lone_handles_share_one_page_of_flags(tmp_path, root):
    run_check(tmp_path, root, "host_flag_check")
