"""The deal of tiles and offsets to the pipelines of the output-stationary forward, checked on the host for every channel pair
(``tests/plans/os_split.cu``)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_deal_holds_its_invariants(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "os_split")
    src = os.path.join(ROOT, "tests", "plans", "os_split.cu")
    build = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe, src], capture_output=True, text=True)
    assert build.returncode == 0, build.stdout + build.stderr
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and " 0 violations" in run.stdout, run.stdout[-2000:]
