"""Builds libdromos_b200.so in-tree with nvcc for sm_100a (the only target), one object per .cu in parallel.

    python -m dromos_b200.build [--force] [--verbose]
"""

from __future__ import annotations

import argparse
import concurrent.futures
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJ = os.path.join(CSRC, "obj")
LIB = os.path.join(HERE, "libdromos_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
CALLS_SRC = os.path.join(CSRC, "calls.cpp")
CALLS = os.path.join(HERE, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))  # the Python callables of abi.Library
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fvisibility=hidden",
         "-I", INCLUDE, "-I", CSRC, "--expt-relaxed-constexpr"]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def headers_mtime():
    times = [os.path.getmtime(os.path.join(CSRC, f)) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    times += [os.path.getmtime(os.path.join(INCLUDE, f)) for f in os.listdir(INCLUDE)]
    return max(times)


def compile_one(src, verbose):
    obj = os.path.join(OBJ, src[:-3] + ".o")
    cmd = [NVCC, *FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    return src, r.returncode, r.stdout + r.stderr


def build_calls(stale):
    """The module of csrc/calls.cpp. Without it abi.Library calls through ctypes, slower and otherwise the same, so a machine without a C++
    compiler or Python's headers gets a warning and the library all the same."""
    if not stale:
        return
    if os.path.exists(CALLS):
        os.remove(CALLS)  # of other sources
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-I", INCLUDE, "-I", sysconfig.get_paths()["include"],
           CALLS_SRC, "-o", CALLS]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        why = r.stdout + r.stderr if r.returncode else None
    except OSError as e:
        why = str(e)
    if why is not None:
        print(f"{why}\nwarning: {os.path.basename(CALLS)} not built (it needs a C++ compiler and Python's headers): calls go through ctypes", file=sys.stderr)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    hdr = headers_mtime()
    todo = []
    for src in sources():
        obj = os.path.join(OBJ, src[:-3] + ".o")
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(hdr, os.path.getmtime(os.path.join(CSRC, src))):
            todo.append(src)
    failed = False
    with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
        for src, rc, out in pool.map(lambda s: compile_one(s, verbose), todo):
            if out.strip() and (verbose or rc != 0):
                print(f"--- {src}\n{out}", file=sys.stderr)
            failed |= rc != 0
    if failed:
        raise RuntimeError("nvcc failed")
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in sources()]
    if todo or not os.path.exists(LIB):
        cmd = [NVCC, "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            print(r.stdout + r.stderr, file=sys.stderr)
            raise RuntimeError("link failed")
    build_calls(force or not os.path.exists(CALLS) or os.path.getmtime(CALLS) < max(hdr, os.path.getmtime(CALLS_SRC)))
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
