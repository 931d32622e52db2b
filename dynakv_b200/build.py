"""Build recipe for the C-ABI library (nvcc, sm_100a only) and the native host side of the Python entry points (g++).

Both are built in-tree, as dynakv_b200/libdynakv_b200.so and dynakv_b200/_host.so (which links to the former); there is
no JIT cache and no other architecture.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libdynakv_b200.so")
HOST = os.path.join(HERE, "_host.so")
HOST_SOURCE = os.path.join(CSRC, "host", "dkv_host.cpp")
HEADER = os.path.join(HERE, "..", "include", "dynakv_b200.h")
SOURCES = ["dkv_api.cu", "dkv_cache.cu", "dkv_generic.cu", "dkv_tiles.cu", "dkv_gate.cu", "dkv_mma_decode.cu", "dkv_short.cu", "dkv_layer.cu", "dkv_project.cu", "dkv_pipe_probe.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--shared", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=default", "-cudart", "shared",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build dynakv_b200")
    return cand


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))] + [HEADER]
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force: bool = False) -> str:
    """The extension that marshals torch tensors into the library's argument structs, against the installed torch."""
    if not force and os.path.exists(HOST) and all(os.path.getmtime(d) <= os.path.getmtime(HOST) for d in (HOST_SOURCE, HEADER)):
        return HOST
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for d in include:
        cmd += ["-isystem", d]
    cmd += [HOST_SOURCE, "-o", HOST, "-L" + HERE, "-l:libdynakv_b200.so", "-L" + os.path.join(root, "lib")]
    cmd += ["-l" + n for n in ("torch_python", "torch", "torch_cpu", "torch_cuda", "c10", "c10_cuda")] + ["-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        build_host()
        return LIB
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + \
          [os.path.join(CSRC, s) for s in SOURCES] + ["-o", LIB]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        sys.stderr.write(res.stderr)
    build_host(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
