"""Builds the CUDA library in-tree: ``sentinel_b200/lib/libsntl_attn.so`` (sm_100a only).

nvcc is invoked directly (one object per ``.cu`` file, then a shared link against the static CUDA
runtime), so the result has no Python or torch dependency and can be bound from C, C++ or ctypes.
Beside it ``sentinel_b200/lib/_sntl_host.so``, the CPython module that puts torch tensors into that ABI (host code only).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libsntl_attn.so")
HOST_MODULE = os.path.join(LIB_DIR, "_sntl_host.so")
HOST_STAMP = os.path.join(LIB_DIR, "_sntl_host.built_for")   # the torch and the Python that the module was built for
OBJ_DIR = os.path.join(HERE, "build")

SOURCES = ["attn_api.cu", "attn_simt_fwd.cu", "attn_simt_bwd.cu", "attn_simt_decode.cu", "attn_f32_fwd_sm100.cu", "attn_f32_bwd_sm100.cu", "attn_f32_route.cu", "layout_convert.cu", "attn_fwd_sm100.cu", "attn_cache_sm100.cu", "attn_bwd_sm100.cu", "attn_dq_sm100.cu",
           "sentinel_compat.cu", "attn_bwd_static_scratch.cu", "ring_nccl.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I", CSRC]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the CUDA library cannot be built")
    return exe


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def host_module_stale() -> bool:
    """Whether the module is older than its source, or was built for another torch or Python than those that run now."""
    import torch
    try:
        with open(HOST_STAMP) as f:
            built_for = f.read()
    except OSError:
        return True
    return built_for != f"{torch.__version__} {sys.version}" or _stale(
        HOST_MODULE, [os.path.join(CSRC, "torch_host.cpp"), os.path.join(ROOT, "include", "sntl_attn.h")])


def build_host_module(force: bool = False) -> str:
    """The CPython module of csrc/torch_host.cpp, against the headers and libraries of the torch that is installed."""
    src = os.path.join(CSRC, "torch_host.cpp")
    if not force and not host_module_stale():
        return HOST_MODULE
    import torch
    from torch.utils import cpp_extension
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    includes = cpp_extension.include_paths() + [sysconfig.get_path("include"), cuda, os.path.join(ROOT, "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DSNTL_TORCH_VERSION="{torch.__version__}"',
           src, "-o", HOST_MODULE] + [x for d in includes for x in ("-isystem", d)]
    cmd += ["-L" + libs, "-Wl,-rpath," + libs, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed on torch_host.cpp")
    with open(HOST_STAMP, "w") as f:
        f.write(f"{torch.__version__} {sys.version}")
    return HOST_MODULE


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".hpp", ".h"))]
    headers.append(os.path.join(ROOT, "include", "sntl_attn.h"))
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        if force or _stale(obj, [os.path.join(CSRC, src)] + headers):
            cmd = [nvcc(), "-c", os.path.join(CSRC, src), "-o", obj] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
            r = subprocess.run(cmd, capture_output=True, text=True)
            if verbose or r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs) + 1)) as ex:
        host = ex.submit(build_host_module, force)
        objs = list(ex.map(compile_one, srcs))
        host.result()
    if force or _stale(LIB, objs):
        cmd = [nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
