"""Builds ``libq4b200.so`` (all CUDA kernels + the C ABI) in-tree with nvcc for sm_100a.

    python -m alpaca_lora_4bit_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  The library is rebuilt when any source under ``csrc/`` or
``include/`` is newer than the ``.so``.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libq4b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    deps.append(os.path.abspath(__file__))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; libq4b200.so cannot be built")
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    objs, procs = [], []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0 or verbose:
            sys.stderr.write(f"--- {os.path.basename(src)} ---\n{out}\n")
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    tmp = LIB + ".tmp"
    subprocess.check_call([nvcc, "-shared", "-o", tmp, *objs, "-Xcompiler", "-fPIC"])
    os.replace(tmp, LIB)
    return LIB


CALL_SRC = os.path.join(CSRC, "host", "q4call.c")
CALL_LIB = os.path.join(PKG, "_q4call.so")


def build_call(force: bool = False) -> str:
    """Builds ``_q4call.so`` (the CPython module that makes the per-token foreign call) with the C compiler."""
    if not force and os.path.exists(CALL_LIB) and os.path.getmtime(CALL_LIB) >= os.path.getmtime(CALL_SRC):
        return CALL_LIB
    import sysconfig
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        raise RuntimeError("no C compiler; _q4call.so cannot be built")
    tmp = CALL_LIB + ".tmp"
    subprocess.check_call([cc, "-O2", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], CALL_SRC, "-o", tmp])
    os.replace(tmp, CALL_LIB)
    return CALL_LIB


TORCH_SRC = os.path.join(CSRC, "host", "q4torch.cpp")
TORCH_LIB = os.path.join(PKG, "_q4torch.so")
TORCH_KEY = os.path.join(PKG, "_q4torch.key")          # what the module beside it was built from


def _torch_call_key() -> str:
    """The sources, and the torch and Python whose binary interface the module is compiled against."""
    import hashlib
    import torch
    h = hashlib.sha256()
    for path in (TORCH_SRC, os.path.join(ROOT, "include", "q4b200.h")):
        with open(path, "rb") as f:
            h.update(f.read())
    return f"{h.hexdigest()} torch {torch.__version__} python {sys.version.split()[0]}\n"


def _torch_call_current(key: str) -> bool:
    try:
        with open(TORCH_KEY) as f:
            return f.read() == key and os.path.exists(TORCH_LIB)
    except OSError:
        return False


def build_torch_call(force: bool = False) -> str:
    """Builds ``_q4torch.so`` (the CPython module that takes torch tensors through the library) with the C++ compiler,
    against the headers and libraries of the installed torch; a module built from other sources or against another torch
    is built again."""
    key = _torch_call_key()
    if not force and _torch_call_current(key):
        return TORCH_LIB
    import sysconfig
    import torch
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("no C++ compiler; _q4torch.so cannot be built")
    base = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    tmp = f"{TORCH_LIB}.{os.getpid()}.tmp"             # (several ranks may find it missing at once)
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                           "-I", os.path.join(base, "include"), "-I", os.path.join(base, "include", "torch", "csrc", "api", "include"),
                           "-I", os.path.join(cuda, "include"), "-I", sysconfig.get_paths()["include"], TORCH_SRC, "-o", tmp,
                           "-L", os.path.join(base, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"])
    os.replace(tmp, TORCH_LIB)
    with open(tmp, "w") as f:
        f.write(key)
    os.replace(tmp, TORCH_KEY)
    return TORCH_LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_call(force="--force" in sys.argv))
    print(build_torch_call(force="--force" in sys.argv))
