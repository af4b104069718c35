"""Builds libflashquest_b200.so (all CUDA kernels + the C ABI) in-tree with nvcc for sm_100a.

    python -m flashquest_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import threading
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libflashquest_b200.so")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
BIND_SRC = os.path.join(CSRC, "fq_bind.cpp")
BIND = os.path.join(LIB_DIR, "_fq_bind.so")       # CPython module over the C ABI (see fq_bind.cpp)
BIND_STAMP = os.path.join(LIB_DIR, "_fq_bind.built_for")       # the torch and the Python it was compiled against

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=default", "--ftz=false", "--prec-div=true",
    "--prec-sqrt=true", "--fmad=true",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def bind_target() -> str:
    """What the CPython module depends on beside its source: torch's C++ ABI, which changes between versions, and Python's."""
    import torch
    return f"torch {torch.__version__} {sys.implementation.cache_tag}"


def bind_built_for() -> str:
    try:
        with open(BIND_STAMP) as f:
            return f.read()
    except OSError:
        return "an unknown torch"


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {what}:\n{r.stdout}\n{r.stderr}")
    if r.stderr:
        print(r.stderr, file=sys.stderr)


def build_bind(force: bool = False, library=lambda: None) -> str:
    """The CPython module: host code only, linked to the running torch and to the library beside it (found through its own
    folder, so the library's symbols stay out of the process).  `library` waits for that library to be linked."""
    target = bind_target()
    if not force and not _stale(BIND, [BIND_SRC, os.path.abspath(__file__), os.path.join(INCLUDE, "flashquest_b200.h")]) and bind_built_for() == target:
        return BIND
    import sysconfig

    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wextra",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(cuda, "include")]
    for inc in ("include", os.path.join("include", "torch", "csrc", "api", "include")):
        cmd += ["-isystem", os.path.join(tdir, inc)]
    obj = BIND[:-3] + ".o"
    _run(cmd + ["-c", BIND_SRC, "-o", obj], BIND_SRC)
    library()
    tlib = os.path.join(tdir, "lib")
    _run(["g++", "-shared", obj, "-o", BIND + ".tmp", "-L", LIB_DIR, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN",
          "-L", tlib, f"-Wl,-rpath,{tlib}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"], BIND)
    os.replace(BIND + ".tmp", BIND)
    with open(BIND_STAMP, "w") as f:
        f.write(target)
    return BIND


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))
    srcs = sources()
    objs = [os.path.join(LIB_DIR, os.path.basename(s)[:-3] + ".o") for s in srcs]
    nvcc = _nvcc()

    def compile_one(pair):
        src, obj = pair
        if not force and not _stale(obj, [src] + headers):
            return None
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-I", INCLUDE, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return r.stderr

    linked = threading.Event()
    bind = ThreadPoolExecutor(max_workers=1).submit(build_bind, force, linked.wait)
    try:
        with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
            logs = list(ex.map(compile_one, zip(srcs, objs)))
        if verbose:
            for log in logs:
                if log:
                    print(log)
        if force or _stale(LIB, objs):
            cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    finally:
        linked.set()
    bind.result()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
