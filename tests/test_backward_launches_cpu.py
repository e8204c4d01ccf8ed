"""What a backward launches, and on how many SMs (no GPU): ``tests/plans/backward_launches.cu`` stands in for the runtime."""
import os
import shutil
import subprocess

import pytest

from fgms_b200 import build as lib_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shares_of_the_sms(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "backward_launches")
    src = os.path.join(ROOT, "tests", "plans", "backward_launches.cu")
    build = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "shared", "-o", exe, src, lib_build.LIB,
                            "-Xlinker", "-rpath," + os.path.dirname(lib_build.LIB)], capture_output=True, text=True)
    assert build.returncode == 0, build.stdout + build.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
