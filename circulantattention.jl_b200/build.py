"""Builds libcircatt_b200.so in-tree with nvcc for sm_100a."""
from __future__ import annotations

import os
import shutil
import subprocess
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
OUT = os.path.join(PKG_DIR, "libcircatt_b200.so")
SOURCES = ["fwd_exact.cu", "fwd_any.cu", "fwd_values_exact.cu", "fwd_values_any.cu", "bwd_exact.cu", "bwd_any.cu", "emit_exact.cu", "emit_any.cu",
           "apply_exact.cu", "apply_any.cu", "operators.cu", "tiled.cu", "pack.cu", "split_pack.cu", "split_fwd.cu", "split_bwd.cu", "line.cu", "api.cu", "static_scratch.cu", "comm.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--use_fast_math", "-Xcompiler", "-fPIC"]


HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_OUT = os.path.join(PKG_DIR, "_circatt_host.so")


def _nvcc():
    return shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _stale():
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    deps.append(os.path.join(PKG_DIR, "..", "include", "circatt_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def _obj_stale(src_path: str, obj: str) -> bool:
    """An object is rebuilt when its own source, any header of csrc/ or the public headers are newer."""
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    inc = os.path.join(PKG_DIR, "..", "include")
    deps = [src_path] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    deps += [os.path.join(inc, f) for f in os.listdir(inc) if f.endswith(".h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    """g++ on the host extension; the ca_* symbols stay undefined and come from the library loaded before it."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], cuda]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"] + ["-I" + d for d in include] +
            [HOST_SRC, "-o", HOST_OUT, "-L" + os.path.join(root, "lib"), "-lc10", "-ltorch", "-ltorch_cpu", "-lc10_cuda",
             "-ltorch_python"])


def _host_stale():
    if not os.path.exists(HOST_OUT):
        return True
    t = os.path.getmtime(HOST_OUT)
    return any(os.path.getmtime(d) > t for d in (HOST_SRC, os.path.join(PKG_DIR, "..", "include", "circatt_b200.h")))


def build(force: bool = False, verbose: bool = False) -> str:
    host = subprocess.Popen(_host_command()) if force or _host_stale() else None
    try:
        return _build_library(force, verbose)
    finally:
        if host is not None and host.wait() != 0:
            raise RuntimeError("g++ failed on host.cpp")


def _build_library(force, verbose):
    if not force and not _stale():
        return OUT
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src[:-3] + ".o")
        objs.append(obj)
        if not force and not _obj_stale(os.path.join(CSRC, src), obj):
            continue
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    subprocess.run([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", OUT, *objs, "-lcudart", "-ldl"], check=True)
    return OUT


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
