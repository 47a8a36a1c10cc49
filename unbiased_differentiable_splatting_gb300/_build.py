"""In-tree build of libuds.so (the CUDA kernels behind the C ABI in include/uds.h).

Each ``csrc/*.cu`` translation unit is compiled for sm_103a in parallel and the
objects are linked into ``libuds.so`` next to this file against the shared CUDA
runtime (the same ``libcudart.so`` torch loads).  ``csrc/uds_torch.cpp`` (the
ops' CUDA kernels and autograd formulas in native code) becomes
``libuds_torch.so``, linked against it and torch.  A rebuild happens only when
a source or header is newer than the library, or, of the second one, when it
was built for another torch or Python.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libuds.so")
OPS_LIB = os.path.join(PKG, "libuds_torch.so")
OPS_SRC = os.path.join(CSRC, "uds_torch.cpp")
OBJ = os.path.join(PKG, "_build")
OPS_STAMP = os.path.join(OBJ, "uds_torch.built_for")
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fno-fast-math"]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libuds.so")


def _sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps():
    return _sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + [os.path.join(ROOT, "include", "uds.h"),
                                                                   os.path.abspath(__file__)]


def _newer(lib, deps) -> bool:
    return os.path.exists(lib) and all(os.path.getmtime(d) <= os.path.getmtime(lib) for d in deps)


def up_to_date() -> bool:
    return _newer(LIB, _deps())


def _ops_target() -> str:
    """What libuds_torch.so is linked against: torch's C++ interface and
    Python's."""
    import torch
    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI') or sys.version}\n"


def ops_built() -> bool:
    """Whether libuds_torch.so is there and was built for this torch and
    Python."""
    try:
        with open(OPS_STAMP) as f:
            return os.path.exists(OPS_LIB) and f.read() == _ops_target()
    except OSError:
        return False


def _ops_up_to_date() -> bool:
    return ops_built() and _newer(OPS_LIB, [OPS_SRC, os.path.join(ROOT, "include", "uds.h"), os.path.abspath(__file__)])


def _torch_dir() -> str:
    import torch
    return os.path.dirname(torch.__file__)


def _ops_compile(obj):
    inc = os.path.join(_torch_dir(), "include")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    return [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-c", OPS_SRC, "-o", obj, "-isystem", inc,
            "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"), "-isystem",
            os.path.join(cuda, "include"), "-isystem", sysconfig.get_path("include")]


def _ops_link(obj, out):
    lib = os.path.join(_torch_dir(), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    return [shutil.which("g++") or "g++", "-shared", "-o", out, obj, LIB, "-L" + lib, "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_python", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN",
            "-Wl,-rpath," + lib]


def _link(cmd, lib):
    tmp = lib + ".tmp"
    r = subprocess.run(cmd(tmp), stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    if r.returncode != 0:
        raise RuntimeError(f"{os.path.basename(lib)} link failed:\n" + r.stdout.decode(errors="replace"))
    os.replace(tmp, lib)


def build(force: bool = False, verbose: bool = False) -> str:
    kernels = force or not up_to_date()
    ops = force or not _ops_up_to_date()
    if not kernels and not ops:
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    procs = []
    objs = []
    ops_obj = os.path.join(OBJ, "uds_torch.o")
    todo = [(OPS_SRC, _ops_compile(ops_obj))] if ops else []
    if kernels:
        nvcc = _nvcc()
        for src in _sources():
            obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
            objs.append(obj)
            todo.append((src, [nvcc, *FLAGS, *ARCH, "-c", src, "-o", obj]))
    for src, cmd in todo:
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    errors = []
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            errors.append(f"{os.path.basename(src)}:\n{out.decode(errors='replace')}")
    if errors:
        raise RuntimeError("libuds.so build failed:\n" + "\n".join(errors))
    if kernels:
        _link(lambda tmp: [nvcc, *ARCH, "-shared", "-cudart", "shared", "-o", tmp, *objs, "-Xlinker",
                           "-rpath,/usr/local/cuda/lib64", "-Xlinker", "-soname,libuds.so"], LIB)
    if ops:
        _link(lambda tmp: _ops_link(ops_obj, tmp), OPS_LIB)
        with open(OPS_STAMP, "w") as f:
            f.write(_ops_target())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
