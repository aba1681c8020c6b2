"""Builds libsphkv_b200.so (sm_100a) with nvcc and the host module host_tables.*.so with g++, in-tree.  No GPU is
needed to build."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_PATH = os.path.join(HERE, "libsphkv_b200.so")
SOURCES = ["capi.cu", "decode.cu", "encode.cu", "lists.cu", "compat.cu", "pool.cu", "kmeans.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; libsphkv_b200.so cannot be built")
    return cand


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_path() -> str:
    import importlib.util
    spec = importlib.util.spec_from_file_location("sphkv_lib_paths", os.path.join(HERE, "_lib.py"))
    lib = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(lib)
    return lib.host_path()


def _host_module(force: bool) -> "subprocess.Popen | None":
    """Starts the compilation of csrc/host_tables.cpp against the installed torch and Python."""
    import sysconfig

    import torch
    src = os.path.join(CSRC, "host_tables.cpp")
    target = _host_path()
    if not (force or _stale(target, [src, os.path.abspath(__file__)])):
        return None
    root = os.path.dirname(torch.__file__)
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-isystem", sysconfig.get_paths()["include"], src, "-o", target,
           "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ and link the shared library, and the host module.  Returns the library's path."""
    nvcc = _nvcc()
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(INCLUDE, "sphkv.h"))
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    objs = []
    procs = []
    host = _host_module(force)
    if host is not None:
        procs.append(("host_tables.cpp", host))
    for src in SOURCES:
        sp = os.path.join(CSRC, src)
        if not os.path.exists(sp):
            continue
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [sp] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", sp, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), flush=True)
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stdout.write(out.decode())
        if pr.returncode != 0:
            raise RuntimeError(f"compilation of {src} failed")
    if force or _stale(LIB_PATH, objs):
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        subprocess.check_call(cmd)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
