"""Ahead-of-time build of the CUDA library (sm_100a only, no JIT, no fallback) and of the native host
path that drives it.

    python -m s2cnn_b200.build            # builds s2cnn_b200/lib/{libs2cnn_b200,s2cnn_host_ops}.so

Replaces the reference's run-time NVRTC path (s2cnn/utils/cuda.py:19-27): kernels are compiled
once with nvcc for the B200 and loaded through the C ABI declared in include/s2cnn_b200.h.
"""
import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(PKG, "csrc", "lib.cu")
PARTS_SRC = os.path.join(PKG, "csrc", "parts.cu")
N_PARTS = 18
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libs2cnn_b200.so")

HOST_SRC = os.path.join(PKG, "host", "host_ops.cpp")
HOST_NAME = "s2cnn_host_ops"
HOST_PATH = os.path.join(LIB_DIR, HOST_NAME + ".so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _sources():
    d = os.path.join(PKG, "csrc")
    return [os.path.join(d, f) for f in sorted(os.listdir(d))] + \
        [os.path.join(os.path.dirname(PKG), "include", "s2cnn_b200.h")]


def _older(path, sources):
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(s) > t for s in sources)


def is_stale():
    return _older(LIB_PATH, _sources())


def build_host(force=False):
    """Compile the native host path (checks, allocation, autograd rules: host/host_ops.cpp) against
    the installed torch if it is missing or older than its source; returns its path."""
    if not force and not _older(HOST_PATH, [HOST_SRC, os.path.join(os.path.dirname(PKG), "include", "s2cnn_b200.h")]):
        return HOST_PATH
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    os.makedirs(LIB_DIR, exist_ok=True)
    tmp = HOST_PATH + ".tmp%d" % os.getpid()
    cmd = ["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=" + HOST_NAME,
           "-DTORCH_API_INCLUDE_EXTENSION_H"] + ["-isystem" + i for i in inc] + [HOST_SRC, "-o", tmp,
           "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda", "-ldl"]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        raise RuntimeError("host path build failed:\n" + res.stdout)
    os.replace(tmp, HOST_PATH)
    return HOST_PATH


def build(force=False, verbose=False):
    """Compile the library and the host path if they are missing or older than their sources;
    returns the library's path."""
    build_host(force)
    if not force and not is_stale():
        return LIB_PATH
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build libs2cnn_b200.so")
    os.makedirs(LIB_DIR, exist_ok=True)
    flags = NVCC_FLAGS + ["-DS2C_SPLIT"] + (["-Xptxas", "-v"] if verbose else [])

    def run(cmd):
        res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if verbose:
            print(res.stdout)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + res.stdout)

    # one object per part (the kernels with many instantiations) beside lib.cu, compiled side by side
    # (nvcc's own -split-compile gave 5 % slower kernels)
    with tempfile.TemporaryDirectory(dir=LIB_DIR) as tmp:
        jobs = [(PARTS_SRC, ["-DS2C_PART=%d" % k], os.path.join(tmp, "part%d.o" % k)) for k in range(N_PARTS)]
        jobs.append((SRC, [], os.path.join(tmp, "lib.o")))
        with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
            list(pool.map(lambda j: run([nvcc] + flags + j[1] + ["-c", j[0], "-o", j[2]]), jobs))
        out = os.path.join(tmp, "lib.so")
        run([nvcc] + NVCC_FLAGS + ["-shared", "-o", out] + [j[2] for j in jobs])
        os.replace(out, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
