"""Builds libmatchattn_b200.so for sm_100a, in-tree, with nvcc alone, and the host extension on top of it with g++.

    python -m matchattention_b200.build [--force]

The translation units (C ABI, one per element type, the built-in scratch area) are compiled in
parallel and linked into matchattention_b200/lib/libmatchattn_b200.so.  The
library carries its own static CUDA runtime and has no Python or torch
dependency; the host extension (csrc/host_binding.cpp, the eager entry points of
ops.py) is compiled against the headers of the running Python and torch and links
to it.  Its file name carries both versions: another Python or torch needs, and
finds missing, a build of its own.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
OBJ_DIR = os.path.join(PKG, "build")
LIB_PATH = os.path.join(LIB_DIR, "libmatchattn_b200.so")
HOST_SOURCE = os.path.join(CSRC, "host_binding.cpp")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")

SOURCES = ["matchattn_api.cu", "matchattn_f32.cu", "matchattn_f16.cu", "matchattn_bf16.cu",
           "matchattn_static_scratch.cu", "matchattn_upsample.cu", "matchattn_volume.cu", "matchattn_field_ops.cu", "matchattn_flow_init.cu", "matchattn_backward.cu"]
HEADERS = ["matchattn_kernels.cuh", "matchattn_lanes.cuh", "matchattn_launch.inl", "matchattn_mma.cuh", "matchattn_binned.cuh",
           "matchattn_staged.cuh"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC,-fvisibility=hidden", "-Xptxas", "-v"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA extension cannot be built on this machine")
    return exe


def host_path() -> str:
    """Where the host extension for the running Python and torch lies."""
    import torch
    return os.path.join(LIB_DIR, f"_host.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so")


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(INCLUDE, "matchattn.h")]
    return any(os.path.getmtime(d) > built for d in deps)


def _build_host() -> None:
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    include = [sysconfig.get_paths()["include"], os.path.join(root, "include"),
               os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{d}" for d in include], HOST_SOURCE,
           "-o", host_path(), f"-L{LIB_DIR}", "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN",
           "-L" + os.path.join(root, "lib"), "-lc10", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on {HOST_SOURCE}:\n{res.stdout}\n{res.stderr}")


def _host_stale() -> bool:
    deps = (HOST_SOURCE, os.path.join(INCLUDE, "matchattn.h"))
    path = host_path()
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _compile(src: str) -> tuple[str, str]:
    obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
    extra = os.environ.get("MATCHATTN_NVCC_EXTRA", "").split()      # e.g. -DMATCHATTN_FAST_EXP=1 for experiments
    cmd = [_nvcc(), *NVCC_FLAGS, *extra, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
    return obj, res.stderr


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _stale():
        _build_library(verbose)
    if force or _host_stale():
        _build_host()
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    with concurrent.futures.ThreadPoolExecutor(max_workers=len(SOURCES)) as pool:
        results = list(pool.map(_compile, SOURCES))
    log = "\n".join(r[1] for r in results)
    with open(os.path.join(OBJ_DIR, "ptxas.log"), "w") as f:
        f.write(log)
    if verbose:
        print(log)
    cmd = [_nvcc(), "-shared", "-o", LIB_PATH, *[r[0] for r in results], "-cudart", "static"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
