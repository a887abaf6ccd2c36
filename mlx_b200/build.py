"""Builds libb200q.so (the C-ABI library) for sm_100a with nvcc, in-tree.

Each .cu file is compiled to an object in mlx_b200/_obj/ (in parallel, rebuilt only
when the source or a header is newer) and linked into mlx_b200/libb200q.so.  nvcc
cross-compiles without a GPU, so this runs anywhere the CUDA toolkit is installed.
csrc/front.cpp becomes the Python extension mlx_b200/_front.so (g++ against torch's headers).

    python -m mlx_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_obj")
LIB = os.path.join(HERE, "libb200q.so")
FRONT = os.path.join(HERE, "_front.so")   # Python extension over LIB (csrc/front.cpp)
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [*os.environ.get("B200Q_EXTRA_NVCC", "").split(),
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "-I", INCLUDE,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libb200q.so")
    return exe


def sources() -> list[str]:
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newest_header() -> float:
    t = 0.0
    for d in (CSRC, INCLUDE):
        for f in os.listdir(d):
            if f.endswith((".h", ".cuh")):
                t = max(t, os.path.getmtime(os.path.join(d, f)))
    return t


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ, src[:-3] + ".o")
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    log = res.stdout + res.stderr
    with open(obj + ".log", "w") as fh:
        fh.write(log)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{log[-4000:]}")
    if verbose:
        print(log)
    return obj


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    hdr = _newest_header()
    todo, objs = [], []
    for src in sources():
        obj = os.path.join(OBJ, src[:-3] + ".o")
        objs.append(obj)
        stamp = max(os.path.getmtime(os.path.join(CSRC, src)), hdr)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < stamp:
            todo.append(src)
    if todo:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(todo))) as ex:
            list(ex.map(lambda s: _compile(s, verbose), todo))
    if todo or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n" + res.stdout + res.stderr)
    front_src = os.path.join(CSRC, "front.cpp")
    if force or not os.path.exists(FRONT) or os.path.getmtime(FRONT) < max(os.path.getmtime(front_src), hdr):
        _build_front(front_src)
    return LIB


def _build_front(src: str) -> None:
    import sysconfig

    from torch.utils import cpp_extension as ce

    inc = [f"-I{p}" for p in (*ce.include_paths(), sysconfig.get_paths()["include"], "/usr/local/cuda/include", INCLUDE)]
    libs = [f"-L{p}" for p in ce.library_paths()] + ["-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", *inc, src, "-o", FRONT, *libs,
           f"-L{HERE}", "-l:libb200q.so", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("building the native front-end failed:\n" + (res.stdout + res.stderr)[-4000:])


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
