"""Build librglru_b200.so (the C-ABI library) in-tree with nvcc for sm_100a, and on top of it _native.so, the eager operators
as native autograd nodes, with the host compiler against the installed PyTorch.

Usage:  python -m griffin_b200.build [--force]

The CUDA library has no dependency on PyTorch; it links the CUDA runtime statically
and resolves the one driver entry point it needs (tensor-map encoding) at run
time.  Object files go to griffin_b200/csrc/_build/.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
SRC_DIR = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(SRC_DIR, "_build")
LIB_PATH = os.path.join(PKG_DIR, "librglru_b200.so")
NATIVE_PATH = os.path.join(PKG_DIR, "_native.so")
SOURCES = ["rglru_scan.cu", "rglru_conv.cu", "rglru_decode.cu", "rglru_gates.cu", "rglru_block.cu", "rglru_fused.cu", "rglru_api.cu", "rglru_noalloc.cu"]
HEADERS = ["rglru_device.cuh", "rglru_scan.cuh", "rglru_tc.cuh", "rglru_vec.cuh", "rglru_mma.cuh", "rglru_internal.h", os.path.join("..", "..", "include", "rglru_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--threads", "2",
]


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found; the RG-LRU kernels cannot be built")
    return found


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile whatever is out of date and return the path of the shared library."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()
    headers = [os.path.join(SRC_DIR, h) for h in HEADERS]
    jobs = []
    objects = []
    for src in SOURCES:
        src_path = os.path.join(SRC_DIR, src)
        obj_path = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        objects.append(obj_path)
        if force or _stale(obj_path, [src_path] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src_path, "-o", obj_path]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
        return res.stderr

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        logs = list(pool.map(run, jobs))
    if verbose:
        for log in logs:
            sys.stderr.write(log)
    if force or jobs or _stale(LIB_PATH, objects):
        run([nvcc, "-shared", "-o", LIB_PATH, *objects, "-gencode", "arch=compute_100a,code=sm_100a"])
    return LIB_PATH


def build_native(force: bool = False) -> str:
    """Compile the native forms of the eager operators (csrc/rglru_torch.cpp) against the installed PyTorch and the library
    above, and return the extension module's path."""
    import sysconfig

    import torch

    source, header = os.path.join(SRC_DIR, "rglru_torch.cpp"), os.path.join(PKG_DIR, "..", "include", "rglru_b200.h")
    if not force and not _stale(NATIVE_PATH, [source, header, torch.__file__]):
        return NATIVE_PATH
    root = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], cuda]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{d}" for d in include), source,
           "-o", NATIVE_PATH, "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch",
           "-ltorch_python", "-L" + PKG_DIR, "-l:librglru_b200.so", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    return NATIVE_PATH


if __name__ == "__main__":
    path = build_library(force="--force" in sys.argv, verbose="-v" in sys.argv)
    build_native(force="--force" in sys.argv)
    print(path)
