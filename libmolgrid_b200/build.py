"""Builds liblmg_b200.so (the CUDA kernels and their C ABI) in-tree with nvcc for sm_100a.

Run as ``python -m libmolgrid_b200.build`` or call :func:`build_library`.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liblmg_b200.so")
SOURCES = ["lmg_gridmaker.cu", "lmg_occupancy.cu", "lmg_misc.cu", "lmg_cabi.cu", "lmg_noalloc.cu", "lmg_records.cu"]
HEADERS = ["lmg_device.cuh", "lmg_atoms.cuh", "lmg_launch.h", "lmg_misc.h", os.path.join("..", "..", "include", "lmg_b200.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    # no fused multiply-add in host code either: the host computes GridMaker's constants
    "-Xcompiler", "-fPIC,-ffp-contract=off,-fvisibility=default",
    "--shared", "--threads", "8",
]


def _nvcc():
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def up_to_date():
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS]
    return all(os.path.getmtime(d) <= t for d in deps)


def build_library(force=False, verbose=False):
    """Compile the library if sources are newer than the built file. Returns its path."""
    if not force and up_to_date():
        return LIB
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + \
        [os.path.join(CSRC, s) for s in SOURCES] + ["-o", LIB]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    return LIB


NATIVE_SRCS = [os.path.join(HERE, "cpp", f) for f in ("bindings.cpp", "bindings_objects.cpp", "bindings_fast.cpp")]


def native_module_path():
    import sysconfig
    return os.path.join(HERE, "molgrid_native" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_native_module(force=False):
    """Compile the pybind11 module over the C++ host layer (g++; links liblmg_b200.so by $ORIGIN)."""
    import concurrent.futures
    import pybind11
    import sysconfig
    import tempfile
    import torch
    out = native_module_path()
    headers = os.path.join(HERE, "cpp", "include", "libmolgrid")
    deps = NATIVE_SRCS + [LIB] + [os.path.join(HERE, "cpp", f) for f in ("bindings_common.h", "bindings_fast.h")] + \
        [os.path.join(headers, f) for f in os.listdir(headers)]
    if not force and os.path.exists(out) and all(os.path.getmtime(d) <= os.path.getmtime(out) for d in deps):
        return out
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    troot = os.path.dirname(torch.__file__)
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-pthread",
             "-I" + pybind11.get_include(), "-I" + sysconfig.get_paths()["include"],
             "-I" + os.path.join(HERE, "cpp", "include"), "-I" + os.path.join(HERE, "..", "include"),
             "-I" + os.path.join(cuda, "include")]
    # torch's headers come with their own pybind11: only the file that reads tensors sees them
    torch_flags = ["-isystem", os.path.join(troot, "include"),
                   "-isystem", os.path.join(troot, "include", "torch", "csrc", "api", "include")]

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)

    with tempfile.TemporaryDirectory() as tmp, concurrent.futures.ThreadPoolExecutor() as pool:
        objs = [os.path.join(tmp, os.path.basename(s) + ".o") for s in NATIVE_SRCS]
        list(pool.map(lambda so: run(["g++", "-c"] + flags + (torch_flags if "fast" in so[0] else []) + [so[0], "-o", so[1]]),
                      zip(NATIVE_SRCS, objs)))
        run(["g++", "-shared", "-pthread"] + objs + ["-o", out, "-L" + HERE, "-llmg_b200",
             "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-L" + os.path.join(troot, "lib"), "-ltorch_python",
             "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN", "-Wl,-rpath," + os.path.join(cuda, "lib64"),
             "-Wl,-rpath," + os.path.join(troot, "lib")])
    return out


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_native_module(force="--force" in sys.argv))
