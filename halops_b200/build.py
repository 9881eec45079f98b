"""Builds the C-ABI shared library ``halops_b200/lib/libhalops_b200.so`` in-tree
with nvcc for sm_100a, and beside it, where torch with CUDA and a C++ compiler are
there, the CPython module that the Python entry points call it through.  No GPU is
needed to build."""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libhalops_b200.so")
SOURCES = ("quant.cu", "gemm.cu")
ABI_HEADER = os.path.join(PKG, "..", "include", "halops_b200.h")
FAST_PATH_DEPS = (os.path.join(CSRC, "fast_path.cpp"), ABI_HEADER)
HEADERS = ("common.cuh", "ptx.cuh", "decode.cuh")


try:
    from ._paths import fast_path_file
except ImportError:  # run as a file, for the C ABI alone
    from _paths import fast_path_file


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def cuda_root() -> str:
    return os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))


def _stale(target: str, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def is_stale() -> bool:
    return _stale(LIB_PATH, [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [ABI_HEADER])


def fast_path_is_stale(torch_version: str) -> bool:
    return _stale(fast_path_file(torch_version), FAST_PATH_DEPS)


def _run(cmd, verbose: bool) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + " ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    if verbose:
        sys.stderr.write(proc.stdout + proc.stderr)


def _build_fast_path(force: bool, verbose: bool) -> None:
    compiler = os.environ.get("CXX") or "g++"
    try:
        import torch
    except ImportError:
        torch = None
    if torch is None or torch.version.cuda is None or shutil.which(compiler) is None:
        # the C ABI does not need it, and the Python wrappers do without
        sys.stderr.write("halops_b200: the native front of the Python calls is not built: it needs torch with CUDA and "
                         f"a C++ compiler ({compiler})\n")
        return
    if not force and not fast_path_is_stale(torch.__version__):
        return
    root = os.path.dirname(torch.__file__)
    cuda = cuda_root()
    _run([
        compiler, "-O2", "-std=c++17", "-fPIC", "-shared",
        "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
        "-I" + os.path.join(cuda, "include"), "-I" + sysconfig.get_paths()["include"],
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
        "-o", fast_path_file(torch.__version__), FAST_PATH_DEPS[0],
        "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
    ], verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source for sm_100a and link the shared library, then the CPython module."""
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or is_stale():
        cmd = [
            _nvcc(),
            "-gencode", "arch=compute_100a,code=sm_100a",
            "-O3", "-std=c++17", "-lineinfo",
            "-Xcompiler", "-fPIC",
            "-shared",
            "-o", LIB_PATH,
        ]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        _run(cmd + [os.path.join(CSRC, f) for f in SOURCES], verbose)
    _build_fast_path(force, verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
