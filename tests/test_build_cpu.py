"""The build (no GPU): which library a copy of the extension is bound to, and when the extension is out of date."""
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


def test_another_pytorch_makes_the_extension_out_of_date(monkeypatch):
    lib_build.build()
    assert not lib_build.needs_build()
    monkeypatch.setattr(lib_build.metadata, "version", lambda name: "0.0.1")
    assert lib_build.needs_build()


def test_the_library_is_built_without_pytorch(monkeypatch):
    def missing(name):
        raise lib_build.metadata.PackageNotFoundError(name)
    lib_build.build()
    commands = []
    monkeypatch.setattr(lib_build.metadata, "version", missing)
    monkeypatch.setattr(lib_build, "_run", lambda cmd, what, verbose: commands.append(what))
    assert lib_build.build(force=True) == lib_build.LIB
    assert commands == ["libfgms_b200.so"]
    assert not lib_build.needs_build()
