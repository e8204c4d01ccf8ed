"""The tcgen05 kernels when a wait runs out: weights that do not arrive and a short limit (``tests/plans/wait_limit.cu``).  The
output is left as it was, the kernel says that it gave up, and the next launch is as good as ever."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_writes_nothing(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "wait_limit")
    src = os.path.join(ROOT, "tests", "plans", "wait_limit.cu")
    build = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert build.returncode == 0, build.stdout + build.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
