"""The build (no GPU): which library a copy of the extension is bound to."""
import os
import shutil
import subprocess
import sys

from fgms_b200 import build as lib_build

BOUND = """
import ctypes, sys
import torch
at = lambda path: ctypes.cast(ctypes.CDLL(path).fgms_b200_version, ctypes.c_void_p).value
for d in sys.argv[1:]:
    assert at(d + "/_native.so") == at(d + "/libfgms_b200.so"), d
assert at(sys.argv[1] + "/_native.so") != at(sys.argv[2] + "/_native.so")
"""


def test_every_copy_of_the_extension_calls_the_library_beside_it(tmp_path):
    dirs = [str(tmp_path / d) for d in ("first", "second")]
    for d in dirs:
        os.mkdir(d)
        for f in (lib_build.LIB, lib_build.BINDING):
            shutil.copy(f, d)
    run = subprocess.run([sys.executable, "-c", BOUND, *dirs], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr
