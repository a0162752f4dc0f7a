"""GPU: a pipeline wait of the stage kernel that runs out (tests/wait_expiry.cu).  The kernel ends by itself, sets the
flag that the host reads even if a single lane's wait ran out, writes no ADO it did not finish, and the context stays
usable."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu


def test_expired_wait_flags_the_launch_and_the_warp_leaves_as_a_whole(tmp_path, root):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "wait_expiry"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(root, "dm-heom_b200", "csrc"),
                    "-o", str(exe), os.path.join(root, "tests", "wait_expiry.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout[-2000:]
