"""Builds the C-ABI CUDA library in-tree: ``nnfusion_b200/libnnf_b200.so`` (sm_100a only)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libnnf_b200.so")
HOST_CALLS = os.path.join(PKG, "_host_calls.so")
SOURCES = ["nnf_api.cu", "dq_gemv.cu", "dq_gemv_direct.cu", "dq_stream.cu", "dq_gemm_tcgen05.cu", "decode_attn.cu", "oneshot_allreduce.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the library cannot be built")


def _older(target: str, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _stale() -> bool:
    return _older(LIB, [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f != "host_calls.cpp"] +
                  [os.path.join(ROOT, "include", "nnf_b200.h")])


def build_host_calls(force: bool = False) -> str:
    """Compile the CPython extension behind repeated calls (host code only, against torch's headers)."""
    src, header = os.path.join(CSRC, "host_calls.cpp"), os.path.join(ROOT, "include", "nnf_b200.h")
    if not force and not _older(HOST_CALLS, [src, header]):
        return HOST_CALLS
    import sysconfig

    from torch.utils import cpp_extension
    inc = [os.path.join(ROOT, "include"), sysconfig.get_paths()["include"], *cpp_extension.include_paths("cuda")]
    lib = [p for p in cpp_extension.library_paths() if os.path.isdir(p)]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           *(f"-I{p}" for p in inc), src, "-o", HOST_CALLS, *(f"-L{p}" for p in lib),
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on host_calls.cpp:\n{r.stdout}")
    return HOST_CALLS


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source for sm_100a into one shared library, and the host extension; returns the former's
    path."""
    build_host_calls(force)
    if not force and not _stale():
        return LIB
    objs = []
    build_dir = os.path.join(PKG, "build")
    os.makedirs(build_dir, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"),
               "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    link = [_nvcc(), "-shared", "-o", LIB, *objs, "-lcudart", "-lcuda"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
