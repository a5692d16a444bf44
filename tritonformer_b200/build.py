"""Builds libtritonformer_b200.so (sm_100a only) from csrc/ with nvcc, and the native host path _host.so from
csrc/host/ with the C++ compiler against this interpreter's torch, in-tree.

    python tritonformer_b200/build.py [--force]

Objects are rebuilt when their source (or any header) is newer.  nvcc cross-compiles
without a GPU, so this runs on a build host as well as on the B200 box.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
HOST = os.path.join(CSRC, "host")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libtritonformer_b200.so")
HOST_LIB = os.path.join(HERE, "_host.so")
CXX = os.environ.get("CXX", "g++")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xcudafe", "--diag_suppress=177",
    # relocatable device code: every translation unit shares ONE device-side status word (status.cu)
    "-rdc=true",
]
# kernels whose warpgroups share out registers: ptxas ignores setmaxnreg in relocatable code
WHOLE = ("attn_bwd_tc05.cu", "attn_bwd128_tc05.cu")


def _sources():
    kernels = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith(".cu")]
    host = [os.path.join(HOST, f) for f in sorted(os.listdir(HOST)) if f.endswith(".cpp")]
    return host + kernels  # the host files take longest to compile


def _headers_mtime(folder):
    m = os.path.getmtime(os.path.join(HERE, "..", "include", "tritonformer_b200.h"))
    for f in os.listdir(folder):
        if f.endswith((".cuh", ".h")):
            m = max(m, os.path.getmtime(os.path.join(folder, f)))
    return m


def _host_flags():
    import torch
    from torch.utils.cpp_extension import include_paths
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(NVCC)))
    inc = include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w",
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)] + ["-I" + i for i in inc]


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("%s failed:\n%s\n%s" % (what, r.stdout, r.stderr))


def _compile(path, force, host_flags):
    src = os.path.basename(path)
    is_host = src.endswith(".cpp")
    obj = os.path.join(OBJ, ("host_" if is_host else "") + os.path.splitext(src)[0] + ".o")
    newest = max(os.path.getmtime(path), _headers_mtime(os.path.dirname(path)))
    if not force and os.path.exists(obj) and os.path.getmtime(obj) > newest:
        return obj
    flags = [f for f in FLAGS if f != "-rdc=true" or src not in WHOLE]
    _run(([CXX] + host_flags if is_host else [NVCC] + flags) + ["-c", path, "-o", obj], "compiling " + src)
    return obj


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    import torch
    host_flags = _host_flags()
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as ex:
        res = list(ex.map(lambda s: _compile(s, force, host_flags), _sources()))
    host = [o for o in res if os.path.basename(o).startswith("host_")]
    kern = [o for o in res if not os.path.basename(o).startswith("host_")]

    def stale(lib, objs):
        return force or not os.path.exists(lib) or os.path.getmtime(lib) < max(os.path.getmtime(o) for o in objs)

    if stale(LIB, kern):
        # nvcc as the linker driver also runs the device link step that -rdc objects need
        _run([NVCC, "-shared", "-o", LIB] + kern
             + ["-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC"], "linking " + LIB)
        if verbose:
            print("linked", LIB)
    if stale(HOST_LIB, host):
        torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
        # the CUDA runtime that libtorch_cuda loads is the one this module uses as well
        _run([CXX, "-shared", "-o", HOST_LIB] + host
             + ["-L" + HERE, "-l:" + os.path.basename(LIB), "-L" + torch_lib, "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
                "-Wl,-rpath,$ORIGIN"], "linking " + HOST_LIB)
        if verbose:
            print("linked", HOST_LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
