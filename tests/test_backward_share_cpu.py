"""The share of the SMs that either pass of a backward gets, checked on the host for every channel pair
(``tests/plans/backward_share.cu``)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shares_hold_their_invariants(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "backward_share")
    src = os.path.join(ROOT, "tests", "plans", "backward_share.cu")
    build = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert build.returncode == 0, build.stdout + build.stderr
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and " 0 violations" in run.stdout, run.stdout[-2000:]
