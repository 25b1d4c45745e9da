"""Build libtpf_b200.so in-tree with nvcc for sm_100a, and the torch extension module `_native` with g++.

    python -m openfold3_triangle_kernel_b200.build [--force] [--verbose]

Each .cu under csrc/ is compiled to an object (in parallel) and linked into
one shared library next to this file.  Nothing is linked against libcuda: the
only driver call (TMA descriptor encoding) is resolved at run time.  The .cpp files
under csrc/ (the eager host path of the operators: checks, allocation, launches, autograd
nodes) become the Python module `_native`, linked against that library and torch.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libtpf_b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
    "-Xcudafe", "--diag_suppress=177",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libtpf_b200.so")
    return exe


def _sources(ext=".cu"):
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(ext))


NATIVE = os.path.join(HERE, "_native" + sysconfig.get_config_var("EXT_SUFFIX"))


def _torch_flags():
    """(compile flags, link flags) of a torch extension, without torch's own build driver."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cflags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wno-unknown-pragmas",
              "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
              "-DTORCH_EXTENSION_NAME=_native"] + ["-isystem" + d for d in inc]
    lib = os.path.join(root, "lib")
    ldflags = ["-L" + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
               "-Wl,-rpath," + lib, "-L" + HERE, "-ltpf_b200", "-Wl,-rpath,$ORIGIN"]
    return cflags, ldflags


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(os.path.dirname(HERE), "include", "tpf_b200.h"))
    return hs


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    hdrs = _headers()
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + hdrs):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
            jobs.append(cmd)
    cflags, ldflags = _torch_flags()
    native_objs = []
    for src in _sources(".cpp"):
        obj = os.path.join(OBJ, os.path.basename(src)[:-4] + ".o")
        native_objs.append(obj)
        if force or _stale(obj, [src] + hdrs):
            jobs.append(["g++"] + cflags + ["-c", src, "-o", obj])

    def run(cmd):
        p = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, p.returncode, p.stdout + p.stderr

    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for cmd, rc, out in ex.map(run, jobs):
                if verbose or rc:
                    sys.stderr.write(" ".join(cmd) + "\n" + out + "\n")
                if rc:
                    raise RuntimeError("compilation failed for " + cmd[-3])
    links = []
    if force or _stale(LIB, objs):
        links.append([nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    if force or links or _stale(NATIVE, native_objs + [LIB]):
        links.append(["g++", "-shared", "-o", NATIVE] + native_objs + ldflags)
    for cmd in links:
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode:
            sys.stderr.write(p.stdout + p.stderr)
            raise RuntimeError("link failed: " + cmd[3])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
