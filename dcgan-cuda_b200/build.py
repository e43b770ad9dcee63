"""Builds libdcgan_b200.so from csrc/*.cu with nvcc for sm_100a, in-tree, and _binding.so next to it.

One nvcc invocation per translation unit (run in parallel), objects cached by
modification time under csrc/build/, then one link step.  No GPU is needed:
nvcc cross-compiles.  _binding.so (csrc/torch_binding.cpp, g++) is the Python
module through which functional.py calls the library on torch tensors.

Run: ``python dcgan-cuda_b200/build.py [--force] [--verbose]``

``DCG_BUILD_FLAGS`` (environment) adds nvcc flags, e.g. ``-DDCG_TC_TRACING`` for the build with the
convolution kernel's timeline and loads-only / MMAs-only switches (``DCG_TC_DEBUG``); use --force with it.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libdcgan_b200.so")
BINDING_SRC = os.path.join(CSRC, "torch_binding.cpp")
BINDING = os.path.join(HERE, "_binding.so")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
CFLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
          "-I", os.path.join(ROOT, "include"), "-I", CSRC] + os.environ.get("DCG_BUILD_FLAGS", "").split()


def _deps():
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))


def _compile(src, force, verbose):
    obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
    newest = max(os.path.getmtime(p) for p in [src] + _deps())
    if not force and os.path.exists(obj) and os.path.getmtime(obj) >= newest:
        return obj
    cmd = [NVCC] + ARCH + CFLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed on " + src)
    return obj


def build(force=False, verbose=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    with concurrent.futures.ThreadPoolExecutor(max_workers=8) as ex:
        objs = list(ex.map(lambda s: _compile(s, force, verbose), srcs))
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        # The CUDA runtime is linked statically and the driver API (tensor-map
        # encoding) is resolved at run time through cudaGetDriverEntryPoint, so the
        # library loads on a machine without a driver (symbol checks on CPU boxes).
        cmd = [NVCC] + ARCH + ["-shared", "-o", LIB] + objs
        subprocess.check_call(cmd)
    _build_binding(force)
    return LIB


def _build_binding(force):
    newest = max(os.path.getmtime(p) for p in [BINDING_SRC] + _deps())
    if not force and os.path.exists(BINDING) and os.path.getmtime(BINDING) >= newest:
        return
    import torch
    root = os.path.join(os.path.dirname(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(NVCC))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I", os.path.join(ROOT, "include"), "-I", sysconfig.get_paths()["include"],
           "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-isystem", os.path.join(cuda, "include"), BINDING_SRC, "-o", BINDING,
           "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
           "-L", HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN"]
    subprocess.check_call(cmd)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
