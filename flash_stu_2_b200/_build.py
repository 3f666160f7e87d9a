"""Compile the CUDA sources under csrc/ into libstu_b200.so next to this file (nvcc, sm_100a only), and the extension
module _native (csrc/native.cpp, the host compiler), through which the interpreter calls it.

Every .cu file is compiled to an object of its own (in parallel, re-used while the source and the shared headers
are older than it) and the objects are linked into the shared library; no device symbol crosses a file boundary,
so no relocatable device code is needed."""
import glob
import importlib.util
import os
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libstu_b200.so")
NATIVE_SRC = os.path.join(CSRC, "native.cpp")
NATIVE = os.path.join(HERE, "_native" + sysconfig.get_config_var("EXT_SUFFIX"))
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def headers():
    return sorted(glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h")))


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(p) > t for p in sources() + headers()) or native_stale()


def native_stale() -> bool:
    if not os.path.exists(NATIVE):
        return True
    t = os.path.getmtime(NATIVE)
    # (torch's own classes are on its boundary: another torch than the one that it was built for needs another)
    torch_version = os.path.join(os.path.dirname(importlib.util.find_spec("torch").origin), "version.py")
    return any(os.path.getmtime(p) > t for p in [NATIVE_SRC, torch_version] + glob.glob(os.path.join(HERE, "..", "include", "*.h")))


def build_native() -> str:
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    others = [f"{root}/include", f"{root}/include/torch/csrc/api/include", sysconfig.get_paths()["include"], f"{cuda}/include"]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-Wextra",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in others:   # (their warnings are not ours)
        cmd += ["-isystem", path]
    cmd += ["-o", NATIVE, NATIVE_SRC, f"-L{HERE}", "-l:libstu_b200.so", f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch",
            "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("the host compiler failed on native.cpp:\n" + res.stdout + res.stderr)
    return NATIVE


def _nvcc():
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _compile(src: str, force: bool, verbose: bool):
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    newest = max(os.path.getmtime(p) for p in [src] + headers())
    if not force and os.path.exists(obj) and os.path.getmtime(obj) >= newest:
        return obj, ""
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", "-o", obj, src]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed on {os.path.basename(src)}:\n" + res.stdout + res.stderr)
    return obj, res.stderr


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    srcs = sources()
    with ThreadPoolExecutor(max_workers=min(len(srcs), os.cpu_count() or 4)) as pool:
        results = list(pool.map(lambda s: _compile(s, force, verbose), srcs))
    res = subprocess.run([_nvcc(), "-shared", "-o", LIB] + [o for o, _ in results], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("link failed:\n" + res.stdout + res.stderr)
    if verbose:
        print("".join(log for _, log in results))
    if force or native_stale():
        build_native()
    return LIB


if __name__ == "__main__":
    import sys
    print(build_library(force="--force" in sys.argv, verbose=True))
