"""Builds liblitenn_b200.so (sm_100a only) next to the package with nvcc.

Usage: python -m litenn_b200.csrc.build [--force] [--verbose]
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
SOURCES = ["lnn_runtime.cu", "lnn_eltwise.cu", "lnn_pool.cu", "lnn_reduce.cu", "lnn_move.cu",
           "lnn_tc.cu", "lnn_small.cu", "lnn_fewch.cu", "lnn_direct.cu", "lnn_depthwise.cu", "lnn_nccl.cu"]
HEADERS = ["lnn_common.cuh", "lnn_tc.cuh", "lnn_tc_dev.cuh", os.path.join("..", "..", "include", "litenn_b200.h")]
LIB = os.path.join(PKG, "liblitenn_b200.so")
NATIVE = os.path.join(PKG, "_native.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--fmad=false", "-prec-div=true", "-prec-sqrt=true"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_native(force=False):
    """Compile the CPython extension of the host layer (g++ and the Python headers)."""
    src = os.path.join(HERE, "host_native.cpp")
    if force or _stale(NATIVE, [src]):
        tmp = f"{NATIVE}.{os.getpid()}"
        subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-Wall",
                               "-I" + sysconfig.get_paths()["include"], src, "-o", tmp])
        os.replace(tmp, NATIVE)         # several processes may get here at once
    return NATIVE


def build(force=False, verbose=False):
    """Compile every .cu to an object (only when out of date) and link the shared library."""
    build_native(force)
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    hdrs = [os.path.join(HERE, h) for h in HEADERS]
    objs, procs = [], []
    for src in SOURCES:
        s = os.path.join(HERE, src)
        o = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + hdrs):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if pr.returncode != 0:
            failed = True
            sys.stderr.write(f"--- {src} failed ---\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src} ---\n{out}\n")
    if failed:
        raise RuntimeError("nvcc failed")
    if force or procs or _stale(LIB, objs):
        cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB] + objs + ["-ldl"]
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
