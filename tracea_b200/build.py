"""Ahead-of-time build of libtracea_b200.so (nvcc, sm_100a only) and of its tensor front end for Python, _ops_native.so
(host compiler, against torch's headers). Cross-compiles without a GPU.

This replaces the reference's run-time path NVRTC -> PTX -> cuModuleLoadData
(src/runtime/manager/kernel.rs:123-327): there is no code generation at run time here.
"""
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtracea_b200.so")
SOURCES = [os.path.join(CSRC, "tracea_ffi.cu")]
HEADERS = [os.path.join(CSRC, f) for f in ("conv2d_sm100.cuh", "conv2d_small_sm100.cuh", "conv2d_window_sm100.cuh", "conv2d_rowband_sm100.cuh", "ptx_sm100.cuh", "layout_kernels.cuh")] + [
    os.path.join(HERE, "..", "include", "tracea_b200.h")]

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared", "-cudart", "static",
]

NATIVE = os.path.join(HERE, "_ops_native.so")
NATIVE_SOURCES = [os.path.join(CSRC, "py_ops.cpp")]
NATIVE_HEADERS = [os.path.join(HERE, "..", "include", "tracea_b200.h")]


def _stale(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(p) > t for p in sources)


def needs_build():
    return _stale(LIB, SOURCES + HEADERS) or _stale(NATIVE, NATIVE_SOURCES + NATIVE_HEADERS)


def _run(cmd, what):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("%s failed:\n" % what + res.stdout + res.stderr)
    return res


def _build_native():
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
          "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch.compiled_with_cxx11_abi()),
          "-I" + sysconfig.get_paths()["include"], "-isystem", os.path.join(root, "include"),
          "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
          "-isystem", os.path.join(cuda, "include")] + NATIVE_SOURCES +
         ["-o", NATIVE, "-L" + HERE, "-l:" + os.path.basename(LIB), "-L" + os.path.join(root, "lib"),
          "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"], "c++")


def build(force=False, verbose=False):
    """Compile what is missing or older than its sources, in-tree."""
    if force or _stale(LIB, SOURCES + HEADERS):
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        res = _run([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES, "nvcc")
        if verbose:
            sys.stderr.write(res.stderr)
    if force or _stale(NATIVE, NATIVE_SOURCES + NATIVE_HEADERS):
        _build_native()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
