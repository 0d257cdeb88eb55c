"""Ahead-of-time build of libelsa_b200.so (plain nvcc, sm_100a only, no torch headers) and of _host.so, the native host
path of the Python operators (g++ against the headers of the installed torch).

    python -m elsa_b200.build            # build if sources are newer than the library
    python -m elsa_b200.build --force
    python elsa_b200/build.py --library  # the C library alone: needs nvcc only, neither torch nor Python's headers
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(CSRC, "build")
LIB_PATH = os.path.join(HERE, "libelsa_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_PATH = os.path.join(HERE, "_host.so")
HOST_STAMP = os.path.join(OBJ_DIR, "_host.built_for")
SOURCES = ["api.cu", "phase2.cu", "fold_simt.cu", "bwd_simt.cu", "fold_tc.cu", "fold_tc3.cu", "fold_tcw.cu", "bwd_tc.cu", "bwd_tc3.cu", "bwd_tcw.cu", "win_tc.cu", "peaks.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _newest_source_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    paths.append(os.path.join(os.path.dirname(HERE), "include", "elsa_b200.h"))
    return max(os.path.getmtime(p) for p in paths)


def needs_build() -> bool:
    return not os.path.exists(LIB_PATH) or os.path.getmtime(LIB_PATH) < _newest_source_mtime()


def _host_built_for() -> str:
    """What _host.so depends on beside its sources: torch's C++ interface and Python's."""
    import sysconfig

    import torch
    return f"torch {torch.__version__} {sysconfig.get_config_var('SOABI')}"


def host_needs_build() -> bool:
    newest = max(os.path.getmtime(HOST_SRC), os.path.getmtime(os.path.join(os.path.dirname(HERE), "include", "elsa_b200.h")))
    if not os.path.exists(HOST_PATH) or os.path.getmtime(HOST_PATH) < newest or not os.path.exists(HOST_STAMP):
        return True
    with open(HOST_STAMP) as f:
        return f.read() != _host_built_for()


def build_host() -> None:
    import sysconfig

    import torch
    root = torch.__path__[0]
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    lib = os.path.join(root, "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DELSA_TORCH_VERSION="{torch.__version__}"', *(f"-I{path}" for path in include), HOST_SRC,
           "-o", HOST_PATH, f"-L{lib}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
           f"-Wl,-rpath,{lib}"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for host.cpp:\n{res.stdout}\n{res.stderr}")
    os.makedirs(OBJ_DIR, exist_ok=True)
    with open(HOST_STAMP, "w") as f:
        f.write(_host_built_for())


def build(force: bool = False, verbose: bool = False) -> str:
    """Both files, the C library first: it is there whatever becomes of the host path."""
    path = build_library(force, verbose)
    if force or host_needs_build():
        build_host()
    return path


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc()

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as pool:
        objs = list(pool.map(compile_one, SOURCES))
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB_PATH


if __name__ == "__main__":
    make = build_library if "--library" in sys.argv else build
    print(make(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
