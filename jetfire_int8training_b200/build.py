"""Build the native parts in-tree: the C-ABI CUDA library (libjetfire_b200.so, nvcc for sm_100a) and the operators' host path
(_host_ops.so, a CPython module over libtorch that calls it).

    python -m jetfire_int8training_b200.build [--force]
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libjetfire_b200.so")
HOST = os.path.join(HERE, "_host_ops.so")
SOURCES = ["nonlinear.cu", "gemm.cu", "noalloc.cu", "lm_loss.cu", "optim.cu"]
HOST_SOURCES = ["host_ops.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared", "--threads", "0"]


def _sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def _build_host():
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    cmd = (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
           + [f for d in inc for f in ("-isystem", d)] + [os.path.join(CSRC, s) for s in HOST_SOURCES]
           + ["-o", HOST, LIB, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
              "-Wl,-rpath,$ORIGIN"])
    subprocess.check_call(cmd)


def build(force=False, verbose=False):
    """Compile every CUDA source into one shared library and the host module on top of it.  Returns the library path."""
    header = os.path.join(os.path.dirname(HERE), "include", "jetfire_b200.h")
    cuda_deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f not in HOST_SOURCES] + [header]
    if force or _stale(LIB, cuda_deps):
        nvcc = os.environ.get("NVCC", "nvcc")
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + _sources() + ["-o", LIB, "-Xlinker", "-soname=libjetfire_b200.so"]
        subprocess.check_call(cmd)
    if force or _stale(HOST, [os.path.join(CSRC, f) for f in HOST_SOURCES] + [header]):
        _build_host()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
