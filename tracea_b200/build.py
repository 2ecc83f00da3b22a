"""Ahead-of-time build of libtracea_b200.so (nvcc, sm_100a only) and of its tensor front end for Python, the extension module
_ops_native (host compiler, against torch's headers). Cross-compiles without a GPU. The library needs nothing of Python or
torch: without torch, or with ``--library-only``, it is all that is built.

This replaces the reference's run-time path NVRTC -> PTX -> cuModuleLoadData
(src/runtime/manager/kernel.rs:123-327): there is no code generation at run time here.
"""
import importlib.util
import os
import runpy
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

# The front end fits one interpreter and one build of torch: the first is in its name, the second in the stamp beside it.
NATIVE = os.path.join(HERE, "_ops_native" + sysconfig.get_config_var("EXT_SUFFIX"))
NATIVE_STAMP = os.path.join(HERE, "_ops_native.stamp")
UNTAGGED_NATIVE = os.path.join(HERE, "_ops_native.so")   # a name that every interpreter would import
NATIVE_SOURCES = [os.path.join(CSRC, "py_ops.cpp")]
NATIVE_HEADERS = [os.path.join(HERE, "..", "include", "tracea_b200.h")]


def _stale(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(p) > t for p in sources)


def _torch_build():
    """What the front end has to fit, as the text of its stamp: the interpreter's suffix, torch's version and the commit it
    was built from. None without torch. (Read from torch/version.py: importing torch takes seconds.)"""
    spec = importlib.util.find_spec("torch")
    if spec is None or not spec.submodule_search_locations:
        return None
    version = runpy.run_path(os.path.join(spec.submodule_search_locations[0], "version.py"))
    return "%s torch %s %s\n" % (sysconfig.get_config_var("EXT_SUFFIX"), version["__version__"], version["git_version"])


def _native_stale():
    fits = _torch_build()
    if fits is None:
        return False
    if os.path.exists(UNTAGGED_NATIVE) or not os.path.exists(NATIVE_STAMP):
        return True
    with open(NATIVE_STAMP) as f:
        return f.read() != fits or _stale(NATIVE, NATIVE_SOURCES + NATIVE_HEADERS)


def needs_build():
    return _stale(LIB, SOURCES + HEADERS) or _native_stale()


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
    with open(NATIVE_STAMP, "w") as f:
        f.write(_torch_build())
    if os.path.exists(UNTAGGED_NATIVE):
        os.remove(UNTAGGED_NATIVE)


def build(force=False, verbose=False, library_only=False):
    """Compile what is missing, older than its sources or made for another interpreter or torch, in-tree. The library alone if
    asked to, or where there is no torch."""
    if force or _stale(LIB, SOURCES + HEADERS):
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        res = _run([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + SOURCES, "nvcc")
        if verbose:
            sys.stderr.write(res.stderr)
    if not library_only and _torch_build() is not None and (force or _native_stale()):
        _build_native()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, library_only="--library-only" in sys.argv))
