"""Builds libbf16n_b200.so (host encoder + policy + sm_100a kernels + C ABI) in-tree with nvcc.

    python -m orin_qwen_lossless_b200.build [--force]

nvcc cross-compiles for sm_100a without a GPU; the .so lands beside this file so it travels with the source tree.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libbf16n_b200.so")
INC = os.path.join(os.path.dirname(PKG), "include")

CUDA_SOURCES = ["gemv.cu", "gemv_staged.cu", "gemv_rings.cu", "gemv_parts.cu", "moe.cu", "moe_decode.cu", "prefill.cu", "expand_tiles.cu", "expand_rows.cu", "peer.cu", "fo.cu", "draft.cu", "adapter.cu", "ep_prefill.cu", "capi.cu"]
HOST_SOURCES = ["encode.cpp", "policy.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC,-pthread",
              "-I", INC]
CXX_FLAGS = ["-O3", "-std=c++17", "-fPIC", "-pthread", "-Wall", "-Wextra", "-I", INC]


def _deps() -> list[str]:
    out = [os.path.join(SRC, f) for f in os.listdir(SRC)]
    out += [os.path.join(INC, f) for f in os.listdir(INC) if f.endswith(".h")]
    return out


def _stale(target: str, sources: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in sources)


def _run(cmd: list[str]) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("build failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is out of date and link, the library and the extension module; returns the library path."""
    build_library(force, verbose)
    build_calls(force)
    return LIB


def build_library(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    deps = _deps()
    jobs = []
    for s in CUDA_SOURCES:
        o = os.path.join(OBJ, s + ".o")
        if force or _stale(o, deps):
            jobs.append(["nvcc", *NVCC_FLAGS, "-c", os.path.join(SRC, s), "-o", o])
    for s in HOST_SOURCES:
        o = os.path.join(OBJ, s + ".o")
        if force or _stale(o, deps):
            jobs.append(["g++", *CXX_FLAGS, "-c", os.path.join(SRC, s), "-o", o])
    if verbose and jobs:
        print(f"compiling {len(jobs)} translation units", file=sys.stderr)
    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        list(ex.map(_run, jobs))
    objs = [os.path.join(OBJ, s + ".o") for s in CUDA_SOURCES + HOST_SOURCES]
    if force or jobs or _stale(LIB, objs):
        _run(["nvcc", "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs, "-lpthread"])
    return LIB


def calls_path() -> str:
    """csrc/host_calls.cpp, an extension module over torch's C++ interface: it is bound to the Python and the torch that it was built for, so
    each pair has a file of its own."""
    import torch
    return os.path.join(PKG, f"_calls-{sysconfig.get_config_var('SOABI')}-torch{torch.__version__}.so")


def build_calls(force: bool = False) -> str:
    """The extension module of the calls that the host bounds; linked against the library beside it."""
    src, path = os.path.join(SRC, "host_calls.cpp"), calls_path()
    if force or _stale(path, [src, os.path.join(INC, "bf16n_c.h")]):
        import torch
        root = os.path.dirname(torch.__file__)
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
               os.path.join(cuda, "include")]
        _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
              *(f"-isystem{i}" for i in inc), src, "-o", path, "-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
              "-L" + PKG, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN"])
    return path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
