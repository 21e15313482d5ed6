"""Builds libcinnamon_b200.so (nvcc, sm_100a) and the native host path _host.so (g++) in-tree.

    python -m cinnamon_b200.build [--force] [--verbose]

The library is plain C ABI (include/cinnamon_b200.h) without torch headers; the host path is the torch extension that
kernels.py calls it through.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libcinnamon_b200.so")
SOURCES = ["quant.cu", "gemm.cu", "linear_few.cu", "moe.cu", "moe_train.cu", "route.cu", "sparse_attn.cu", "attn_tc.cu", "indexer.cu", "wgrad.cu", "capi.cu"]
HOST_DIR = os.path.join(CSRC, "host")
HOST_PATH = os.path.join(LIB_DIR, "_host.so")
HOST_SOURCES = ["linear.cpp", "attention.cpp", "moe.cpp", "moe_train.cpp", "module.cpp"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the cinnamon_b200 library cannot be built")
    return exe


def _stale(target: str, *folders: str) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(d, f) for d in folders for f in os.listdir(d)]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "cinnamon_b200.h"))
    return any(os.path.isfile(d) and os.path.getmtime(d) > t for d in deps)


def _host_commands(obj_dir: str):
    """(compile commands by object, link command) of the host path."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{d}" for d in inc)]
    objs = {os.path.join(obj_dir, "host_" + f.replace(".cpp", ".o")): os.path.join(HOST_DIR, f) for f in HOST_SOURCES}
    link = ["g++", "-shared", "-o", HOST_PATH + ".tmp", *objs, "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
    return {o: ["g++", *flags, "-c", src, "-o", o] for o, src in objs.items()}, link


def build(force: bool = False, verbose: bool = False) -> str:
    new_lib = force or _stale(LIB_PATH, CSRC)
    new_host = force or _stale(HOST_PATH, HOST_DIR)
    if not (new_lib or new_host):
        return LIB_PATH
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    jobs = []                                                   # (source, command)
    link, link_host = [], []
    if new_lib:
        nvcc = _nvcc()
        objs = [os.path.join(obj_dir, src.replace(".cu", ".o")) for src in SOURCES]
        extra = ["-Xptxas", "-v"] if verbose else []
        jobs += [(src, [nvcc, *extra, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]) for src, obj in zip(SOURCES, objs)]
        link = [nvcc, "-shared", "-o", LIB_PATH + ".tmp", *objs, "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a"]
    if new_host:
        compiles, link_host = _host_commands(obj_dir)
        jobs += [(cmd[-3], cmd) for cmd in compiles.values()]
    procs = [(src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)) for src, cmd in jobs]
    failed = []
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            print(out)
        if p.returncode != 0:
            failed.append(src)
    if failed:
        raise RuntimeError(f"compilation failed: {', '.join(failed)}")
    for cmd, path in ((link, LIB_PATH), (link_host, HOST_PATH)):
        if cmd:
            subprocess.check_call(cmd)
            os.replace(path + ".tmp", path)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
