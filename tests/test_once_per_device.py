"""The shared-memory limit of the network's kernels is set on every device that runs them, not once per process: the
class that keeps track of it, compiled on its own (one GPU cannot show the second device)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"


def test_a_device_is_pending_until_it_is_set(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not here")
    exe = str(tmp_path / "once")
    r = subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "xmcml_b200", "csrc"), "-I", CUDA,
                        os.path.join(ROOT, "tests", "c_abi", "once_per_device.cpp"), "-o", exe, "-pthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"
