"""In-tree nvcc build of ``libfast_mimi_b200.so`` for sm_100a.

``python -m fast_mimi_b200._build`` (or ``__graft_entry__.build()``) compiles every ``csrc/*.cu`` into
``fast_mimi_b200/lib/libfast_mimi_b200.so`` and ``csrc/bind`` into the extension module ``_fm_bind.so`` beside it.  The library is never built implicitly at import or call
time: a missing library is an error (see ``_native.load``).
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libfast_mimi_b200.so")
BIND_SOURCE = os.path.join(CSRC, "bind", "fm_bind.cpp")
BIND_PATH = os.path.join(LIB_DIR, "_fm_bind.so")      # extension module: the per-call host work

NVCC_FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC"]


def find_nvcc() -> str:
    cand = os.environ.get("FAST_MIMI_B200_NVCC") or shutil.which("nvcc")
    if cand is None:
        home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        cand = os.path.join(home, "bin", "nvcc")
    if not os.path.exists(cand):
        raise RuntimeError(f"nvcc not found (looked at {cand}); set FAST_MIMI_B200_NVCC")
    return cand


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(os.path.dirname(PKG), "include", "*.h"))
    return any(os.path.getmtime(d) > built for d in deps)


def _build_bind() -> None:
    """g++ build of the extension module, linked against the library next to it and against torch."""
    import torch
    from torch.utils import cpp_extension
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    include = [os.path.join(os.path.dirname(find_nvcc()), "..", "include"), *cpp_extension.include_paths(),
               sysconfig.get_paths()["include"]]
    cxx = os.environ.get("CXX") or shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        raise RuntimeError("no C++ compiler found; set CXX")
    tmp = BIND_PATH + ".tmp"
    subprocess.run([cxx, "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                    *("-I" + i for i in include), BIND_SOURCE, "-o", tmp, "-L" + torch_lib, "-ltorch_python", "-ltorch",
                    "-ltorch_cpu", "-lc10", "-lc10_cuda", "-L" + LIB_DIR, "-l:libfast_mimi_b200.so", "-Wl,-rpath,$ORIGIN"],
                   check=True)
    os.replace(tmp, BIND_PATH)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the library and the extension module if a source is newer than them; return the library's path."""
    path = _build_library(force, verbose)
    header = os.path.join(os.path.dirname(PKG), "include", "fast_mimi_b200.h")
    if force or not os.path.exists(BIND_PATH) or max(os.path.getmtime(BIND_SOURCE), os.path.getmtime(header)) > os.path.getmtime(BIND_PATH):
        _build_bind()
    return path


def _build_library(force: bool, verbose: bool) -> str:
    if not force and not _stale():
        return LIB_PATH
    nvcc = find_nvcc()
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    cmds = []
    for src in sources():
        obj = os.path.join(LIB_DIR, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        cmds.append(cmd)
        objs.append(obj)
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:     # one nvcc per source
        list(pool.map(lambda cmd: subprocess.run(cmd, check=True), cmds))
    tmp = LIB_PATH + ".tmp"
    # the link step names the same architecture, so nvcc does not fall back to (and warn about) its default one
    subprocess.run([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", tmp, *objs], check=True)
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
