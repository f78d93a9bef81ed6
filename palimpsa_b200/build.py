"""Build libpalimpsa_b200.so (nvcc, sm_100a) and the torch front end over it (_torch_ops, host C++) in-tree.

    python -m palimpsa_b200.build [--force]

Cross-compiles without a GPU.  The library links the CUDA runtime statically and has no other
dependency (no torch, no Python): its whole surface is the C ABI in include/palimpsa_b200.h.  The front end is a
Python extension module that links torch and the library.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
ROOT = os.path.dirname(PKG)
LIB = os.path.join(PKG, "libpalimpsa_b200.so")
EXT = os.path.join(PKG, "_torch_ops" + sysconfig.get_config_var("EXT_SUFFIX"))
EXT_STAMP = os.path.join(PKG, "_torch_ops.built_for")      # the torch version EXT was compiled and linked against
EXT_SOURCE = os.path.join(CSRC, "torch_ops.cpp")
HEADER = os.path.join(ROOT, "include", "palimpsa_b200.h")
UNITS = ("abi", "fwd", "fwd_tall", "bwd", "decode", "segments", "summary_tc", "carry_tc", "layer", "peer")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--extended-lambda",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _sources():
    out = [HEADER]
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            out.append(os.path.join(CSRC, f))
    return out


def _older(target, sources) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(s) > os.path.getmtime(target) for s in sources)


def _torch_version() -> str:
    from importlib.metadata import version
    return version("torch")


def _ext_is_for_this_torch() -> bool:
    """The front end uses torch's C++ interface, which other versions do not keep."""
    if not os.path.exists(EXT_STAMP):
        return False
    with open(EXT_STAMP) as f:
        return f.read().strip() == _torch_version()


def needs_build() -> bool:
    return _older(LIB, _sources()) or _older(EXT, [HEADER, EXT_SOURCE]) or not _ext_is_for_this_torch()


def _run(cmd, what, log=None):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if log:
        with open(log, "w") as f:
            f.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")


def _compile_ext(obj):
    """The front end's object file: torch's headers, plain host C++."""
    from torch.utils import cpp_extension as E
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [*E.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_torch_ops",
          "-DTORCH_API_INCLUDE_EXTENSION_H", *(f"-I{d}" for d in inc), "-c", EXT_SOURCE, "-o", obj], "g++ on torch_ops.cpp")


def _link_ext(obj):
    import torch
    from torch.utils import cpp_extension as E
    tmp = EXT + ".tmp"
    libs = [f"-L{d}" for d in E.library_paths()]
    _run(["g++", "-shared", "-o", tmp, obj, f"-L{PKG}", "-l:libpalimpsa_b200.so", *libs, "-ltorch", "-ltorch_cpu",
          "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN",
          f"-Wl,-rpath,{os.path.join(os.path.dirname(torch.__file__), 'lib')}"], "link of _torch_ops")
    os.replace(tmp, EXT)
    with open(EXT_STAMP, "w") as f:
        f.write(_torch_version() + "\n")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)

    headers = [s for s in _sources() if not s.endswith(".cu")]

    def compile_unit(u):
        obj = os.path.join(objdir, u + ".o")
        deps = headers + [os.path.join(CSRC, u + ".cu")]
        if not force and os.path.exists(obj) and all(os.path.getmtime(d) <= os.path.getmtime(obj) for d in deps):
            return obj                                # this unit's sources are older than its object
        _run([_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, u + ".cu"), "-o", obj], f"nvcc on {u}.cu",
             os.path.join(objdir, u + ".ptxas.log"))
        return obj

    ext_obj = os.path.join(objdir, "torch_ops.o")
    ext_stale = force or _older(ext_obj, [HEADER, EXT_SOURCE]) or not _ext_is_for_this_torch()
    with ThreadPoolExecutor(len(UNITS) + 1) as ex:
        ext_job = ex.submit(_compile_ext, ext_obj) if ext_stale else None
        objs = list(ex.map(compile_unit, UNITS))
        if ext_job:
            ext_job.result()
    tmp = LIB + ".tmp"
    _run([_nvcc(), "-shared", "-o", tmp, *objs, "-gencode", "arch=compute_100a,code=sm_100a"], "link")
    os.replace(tmp, LIB)
    _link_ext(ext_obj)
    if verbose:
        print("built", LIB, EXT)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
