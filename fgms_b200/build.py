"""Build ``libfgms_b200.so`` (nvcc, sm_100a) and the PyTorch extension ``_native.so`` (g++) in-tree.

    python -m fgms_b200.build [--force] [--verbose]

The library is a plain C-ABI shared object (see ``include/fgms_b200.h``); it links only the CUDA
runtime, not PyTorch.  ``_native.so`` is the PyTorch binding on top of it and finds it beside itself; without PyTorch
the library alone is built.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
import tempfile
from importlib import metadata

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libfgms_b200.so")
SOURCES = [os.path.join(CSRC, "fgms_abi.cu")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    # no GNU-unique symbols: two builds of the library in one process keep their launch state apart
    "-Xcompiler", "-fPIC,-fno-gnu-unique", "-shared", "-cudart", "shared", "-ldl",
]


BINDING = os.path.join(HERE, "_native.so")
BINDING_SOURCE = os.path.join(CSRC, "torch_binding.cpp")
BUILT_FOR = os.path.join(HERE, "_native.built_for")  # the PyTorch and Python that _native.so was built for


def _deps():
    out = list(SOURCES)
    for d in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        out += [os.path.join(d, f) for f in os.listdir(d) if f.endswith((".cuh", ".h", ".cu"))]
    return out


def _stale(target: str, sources) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in sources)


def _host() -> str | None:
    """The PyTorch and Python of this environment; None without PyTorch."""
    try:
        return f"torch {metadata.version('torch')}, {sysconfig.get_config_var('SOABI')}"
    except metadata.PackageNotFoundError:
        return None


def _built_for() -> str | None:
    if not os.path.exists(BUILT_FOR):
        return None
    with open(BUILT_FOR) as f:
        return f.read()


def needs_build() -> bool:
    if _stale(LIB, _deps()):
        return True
    host = _host()
    return host is not None and (_built_for() != host or
                                 _stale(BINDING, [BINDING_SOURCE, os.path.join(os.path.dirname(HERE), "include", "fgms_b200.h")]))


def _run(cmd, what: str, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"building {what} failed")


def _build_binding(verbose: bool) -> None:
    import torch
    from torch.utils import cpp_extension
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    include = cpp_extension.include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd += [f for d in include for f in ("-isystem", d)]
    # The extension names the library by its place beside itself, through a stand-in of that name at link time: under a
    # bare name the loader would hand it the library of another copy that the process has loaded already.
    with tempfile.TemporaryDirectory() as tmp:
        beside = os.path.join(tmp, "beside.so")
        _run(["g++", "-shared", "-fPIC", "-x", "c++", os.devnull, "-o", beside, "-Wl,-soname,$ORIGIN/libfgms_b200.so"], "a stand-in", verbose)
        cmd += [BINDING_SOURCE, "-o", BINDING, "-Wl,--no-as-needed", beside, "-L" + lib_dir, "-ltorch_python", "-ltorch", "-ltorch_cpu",
                "-lc10", "-lc10_cuda", "-Wl,-rpath," + lib_dir]
        _run(cmd, "_native.so", verbose)
    with open(BUILT_FOR, "w") as f:
        f.write(_host())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    _run([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + SOURCES + ["-o", LIB], "libfgms_b200.so", verbose)
    if _host() is None:
        sys.stderr.write("PyTorch is not installed: _native.so is not built\n")
    else:
        _build_binding(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
