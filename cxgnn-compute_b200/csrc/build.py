"""Builds libcxgnn_b200.so from the .cu files in this directory with nvcc for sm_100a, and the Python backend's host
module (native.cpp, g++ against torch's headers) that calls it.

Usage: python build.py [--force] [--verbose]
The library is written next to this file, the module next to the backend; nothing is installed.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libcxgnn_b200.so")
NATIVE_SRC = os.path.join(HERE, "native.cpp")
NATIVE = os.path.join(HERE, "..", "cxgnncomp_backend", "_native.so")
OBJ_DIR = os.path.join(HERE, "build")
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NVCC = os.environ.get("NVCC", os.path.join(CUDA_HOME, "bin", "nvcc"))
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def sources():
    return sorted(f for f in os.listdir(HERE) if f.endswith(".cu"))


def headers():
    inc = os.path.join(HERE, "..", "..", "include")
    hs = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(inc, f) for f in os.listdir(inc) if f.endswith(".h")]
    return hs


def stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def native_command():
    import torch
    from torch.utils.cpp_extension import include_paths
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + ["-I" + p for p in include_paths() + [sysconfig.get_paths()["include"], os.path.join(CUDA_HOME, "include")]]
            + [NATIVE_SRC, "-o", NATIVE, "-L" + libs, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-ldl"])


def build(force=False, verbose=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdrs = headers() + [os.path.abspath(__file__)]
    jobs = []
    objs = []
    for src in sources():
        obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
        objs.append(obj)
        if force or stale(obj, [os.path.join(HERE, src)] + hdrs):
            cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(HERE, src), "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    if force or stale(NATIVE, [NATIVE_SRC] + hdrs):
        jobs.append(native_command())

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("the compiler failed: " + " ".join(cmd))
    if jobs or force or stale(LIB, objs):
        cmd = [NVCC, "-shared", "-o", LIB] + objs
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
