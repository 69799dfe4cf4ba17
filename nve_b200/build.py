"""Build libnve_kernels.so (sm_100a) in-tree with nvcc.

The library is the product: a plain C-ABI shared object with no torch or Python types in its
signatures (see include/nve_kernels.h).  ``python -m nve_b200.build`` compiles every ``.cu`` file
under ``csrc/`` in parallel and links ``nve_b200/lib/libnve_kernels.so``, then builds the Python
module ``nve_b200/_host.so`` (csrc/host/), native wrappers over the library for torch tensors.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_DIR = os.path.join(PKG_DIR, "lib")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(LIB_DIR, "libnve_kernels.so")
HOST_SRC = os.path.join(CSRC, "host", "torch_calls.cpp")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libnve_kernels.so cannot be built")
    return exe


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _digest(path: str, extra: str) -> str:
    h = hashlib.sha256(extra.encode())
    for dep in [path] + [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cuh", ".h"))] + [
        os.path.join(PKG_DIR, "..", "include", "nve_kernels.h")
    ]:
        with open(dep, "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def _compile_one(src: str, verbose: bool, ptxas_v: bool) -> str:
    obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
    flags = list(NVCC_FLAGS) + (["-Xptxas", "-v"] if ptxas_v else [])
    stamp = obj + ".sha"
    dig = _digest(src, " ".join(flags))
    if not ptxas_v and os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == dig:
        return obj
    cmd = [_nvcc()] + flags + ["-c", src, "-o", obj]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
    if ptxas_v or verbose:
        sys.stderr.write(res.stderr)
    with open(stamp, "w") as fh:
        fh.write(dig)
    return obj


def build_host(verbose: bool = False, force: bool = False) -> str:
    """Compile the torch-tensor wrappers against the installed torch; rebuilt when the source, the C ABI or torch changes."""
    import sysconfig

    import torch

    stamp = os.path.join(OBJ_DIR, "_host.sha")
    h = hashlib.sha256(f"{torch.__version__} {sys.version}".encode())
    for dep in (HOST_SRC, os.path.join(PKG_DIR, "..", "include", "nve_kernels.h")):
        with open(dep, "rb") as fh:
            h.update(fh.read())
    if not force and os.path.exists(HOST_PATH) and os.path.exists(stamp) and open(stamp).read() == h.hexdigest():
        return HOST_PATH
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           HOST_SRC, "-o", HOST_PATH]
    for inc in (sysconfig.get_paths()["include"], os.path.join(root, "include"),
                os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")):
        cmd += ["-isystem", inc]
    cmd += ["-L", LIB_DIR, "-lnve_kernels", "-Wl,-rpath,$ORIGIN/lib", "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch_python"]
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{res.stdout}\n{res.stderr}")
    with open(stamp, "w") as fh:
        fh.write(h.hexdigest())
    return HOST_PATH


def build(verbose: bool = False, ptxas_v: bool = False, force: bool = False) -> str:
    """Compile and link the library; returns its path.  Incremental unless ``force``."""
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    if force:
        for f in os.listdir(OBJ_DIR):
            os.remove(os.path.join(OBJ_DIR, f))
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as pool:
        objs = list(pool.map(lambda s: _compile_one(s, verbose, ptxas_v), srcs))
    newest = max(os.path.getmtime(o) for o in objs)
    if force or not os.path.exists(LIB_PATH) or os.path.getmtime(LIB_PATH) < newest:
        cmd = [_nvcc(), "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    build_host(verbose, force)
    return LIB_PATH


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, ptxas_v="--ptxas" in sys.argv, force="--force" in sys.argv))
