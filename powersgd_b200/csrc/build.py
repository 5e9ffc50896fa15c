"""Builds the native library in-tree: `python -m powersgd_b200.csrc.build`.

Every translation unit is compiled for sm_100a only (`-gencode arch=compute_100a,code=sm_100a`)
and linked into `libpsgd_b200.so` next to the sources, with the CUDA runtime linked statically
so that the library loads beside any PyTorch build. nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
import warnings
from typing import List

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libpsgd_b200.so")
OBJ_DIR = os.path.join(HERE, "build")
# the same sources with -DPSGD_BOUNDS_CHECK (see psgd_bounds.cuh): kernels validate their tiles and
# record violations instead of accessing memory; loaded through PSGD_B200_LIB by the checked tests
DEBUG_LIB = os.path.join(HERE, "libpsgd_b200_debug.so")
DEBUG_OBJ_DIR = os.path.join(HERE, "build_debug")
SCAN_LIB = os.path.join(HERE, "_tensor_scan.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fvisibility=hidden", "--use_fast_math=false"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def sources() -> List[str]:
    return sorted(f for f in os.listdir(HERE) if f.endswith((".cu", ".cpp")))


def _digest(paths: List[str]) -> str:
    h = hashlib.sha256()
    for p in sorted(paths):
        with open(p, "rb") as fp:
            h.update(p.encode())
            h.update(fp.read())
    return h.hexdigest()


def _compile_one(nvcc: str, src: str, verbose: bool, debug: bool = False) -> str:
    obj = os.path.join(DEBUG_OBJ_DIR if debug else OBJ_DIR, os.path.splitext(src)[0] + ".o")
    cmd = [nvcc, *ARCH, *[c for c in COMMON if c != "--use_fast_math=false"], "-I", HERE, "-c", os.path.join(HERE, src), "-o", obj]
    if debug:
        cmd.insert(1, "-DPSGD_BOUNDS_CHECK")
    if src.endswith(".cpp"):
        cmd.insert(1, "-x")
        cmd.insert(2, "cu")
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        sys.stderr.write(res.stderr)
    return obj


def scan_target() -> str:
    """What the list checks are compiled for. They have PyTorch's tensor layout compiled in, so another build of
    it must not load them, whether or not it has the symbols that they ask for."""
    import platform

    import torch

    return f"torch {torch.__version__} {torch.version.git_version}, python {platform.python_version()}"


def _build_scan() -> None:
    """The list checks (host/tensor_scan.cpp), a CPython extension for the PyTorch of this interpreter."""
    src = os.path.join(HERE, "host", "tensor_scan.cpp")
    import sysconfig

    import torch

    stamp_path = os.path.join(OBJ_DIR, "scan_stamp.txt")
    stamp = f"{_digest([src])} {scan_target()}"
    if os.path.exists(SCAN_LIB) and os.path.exists(stamp_path):
        with open(stamp_path) as fp:
            if fp.read() == stamp:
                return
    base = os.path.dirname(os.path.abspath(torch.__file__))
    includes = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DPSGD_SCAN_TARGET="{scan_target()}"',
           *[f"-isystem{i}" for i in includes], src, "-o", SCAN_LIB,
           f"-L{os.path.join(base, 'lib')}", "-lc10", "-ltorch_cpu", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on {src}:\n{res.stdout}\n{res.stderr}")
    with open(stamp_path, "w") as fp:
        fp.write(stamp)


def build(force: bool = False, verbose: bool = False, debug: bool = False) -> str:
    """`debug=True` builds the bounds-checked variant (libpsgd_b200_debug.so) instead."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    try:
        _build_scan()
    except Exception as exc:   # no PyTorch, headers of Python or host compiler: the package asks in Python instead, more slowly
        if os.path.exists(SCAN_LIB):
            os.remove(SCAN_LIB)
        warnings.warn(f"list checks not built ({exc})", stacklevel=2)
    srcs = sources()
    headers = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".h", ".cuh"))]
    obj_dir, lib = (DEBUG_OBJ_DIR, DEBUG_LIB) if debug else (OBJ_DIR, LIB)
    stamp_path = os.path.join(obj_dir, "stamp.txt")
    digest = _digest([os.path.join(HERE, s) for s in srcs] + headers)
    if not force and os.path.exists(lib) and os.path.exists(stamp_path):
        with open(stamp_path) as fp:
            if fp.read().strip() == digest:
                return lib
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as pool:
        objs = list(pool.map(lambda s: _compile_one(nvcc, s, verbose, debug), srcs))
    link = [nvcc, *ARCH, "-shared", "-cudart", "static", "-o", lib, *objs, "-lpthread", "-ldl", "-lrt"]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    with open(stamp_path, "w") as fp:
        fp.write(digest)
    return lib


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv, debug="--debug" in sys.argv)
    print(path)
