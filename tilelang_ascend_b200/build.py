"""Build libqgemm.so (the C-ABI shared library, nvcc for sm_100a) and the extension module _qhost (the operators' native
call path, g++ against torch's headers) in-tree.

    python -m tilelang_ascend_b200.build [--force] [--verbose]

Both land next to this file; each is rebuilt when one of its sources under ``csrc/`` or ``include/qgemm.h`` is newer
than it.  The extension's file name carries the interpreter and the torch it was compiled against, so that it is built
again, and never loaded, under another one.  A finished file takes its place in one step: a process that loads it while
another one builds sees the old or the new file, never a half-written one.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libqgemm.so")
HOST_SOURCE = os.path.join(CSRC, "host.cpp")
SOURCES = ["qgemm_api.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared",
]


def host_lib() -> str:
    """Where the extension module for this interpreter and this torch belongs."""
    import sysconfig

    import torch
    abi = "" if torch._C._GLIBCXX_USE_CXX11_ABI else ".oldabi"
    return os.path.join(PKG, f"_qhost.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}{abi}.so")


def _deps():
    deps = [os.path.join(ROOT, "include", "qgemm.h")]
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            deps.append(os.path.join(CSRC, f))
    return deps


def _stale(target, deps) -> bool:
    if not os.path.isfile(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _lib_stale() -> bool:
    return _stale(LIB, _deps())


def _host_stale() -> bool:
    return _stale(host_lib(), [os.path.join(ROOT, "include", "qgemm.h"), HOST_SOURCE])


def needs_build() -> bool:
    return _lib_stale() or _host_stale()


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.isfile(cand):
            return cand
    raise RuntimeError("nvcc not found; libqgemm.so cannot be built")


def _compile(cmd, target, verbose):
    """Run the command with a temporary output file, which then takes the target's place."""
    tmp = f"{target}.{os.getpid()}.tmp"
    try:
        _run([*cmd, "-o", tmp], verbose)
        os.replace(tmp, target)
    finally:
        if os.path.exists(tmp):
            os.remove(tmp)


def _run(cmd, verbose):
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout)
    if res.returncode != 0:
        raise RuntimeError("build failed:\n" + " ".join(cmd))


def _host_command():
    import sysconfig

    import torch
    base = os.path.dirname(torch.__file__)
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(find_nvcc())), "include")]
    lib = os.path.join(base, "lib")
    return ([os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-Wextra",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [x for d in inc for x in ("-isystem", d)]  # (warnings for this module's own code only)
            + [HOST_SOURCE, f"-L{lib}", f"-Wl,-rpath,{lib}", "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda",
               "-lc10", "-lc10_cuda"])


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _lib_stale():
        cmd = [find_nvcc(), *NVCC_FLAGS]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        _compile(cmd + [os.path.join(CSRC, s) for s in SOURCES], LIB, verbose)
    if force or _host_stale():
        _compile(_host_command(), host_lib(), verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
