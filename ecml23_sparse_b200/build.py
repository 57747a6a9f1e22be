"""Builds, in-tree, the CUDA library ``libffi_b200.so`` for sm_100a with nvcc and ``_native.so``, the
binding of its hot entry points over torch tensors, with the host compiler.

``python -m ecml23_sparse_b200.build`` or :func:`build`.  Each is rebuilt when a source file is newer
than it, the binding also when it was built for another torch.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB_PATH = os.path.join(PKG_DIR, "libffi_b200.so")
BINDING_SRC = os.path.join(CSRC, "binding.cpp")
BINDING_PATH = os.path.join(PKG_DIR, "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=default",
]


class CompilerMissing(RuntimeError):
    """This machine has no compiler; what was built elsewhere may be used."""


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise CompilerMissing("nvcc not found; the FFI library cannot be built")
    return exe


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


OBJ_DIR = os.path.join(PKG_DIR, "build")


def _compile_one(args) -> str:
    src, obj, extra, verbose = args
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", "-I", INCLUDE, "-I", CSRC, *extra, src, "-o", obj]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return obj


def build(force: bool = False, verbose: bool = False, extra: list[str] | None = None) -> str:
    """Compiles every source file to an object (in parallel; an object is reused while it is newer than
    its source and the shared headers) and links them into the shared library."""
    if not force and not _stale():
        return LIB_PATH
    from concurrent.futures import ThreadPoolExecutor

    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(INCLUDE, "*.h"))
    newest_header = max((os.path.getmtime(h) for h in headers), default=0.0)
    jobs, objs = [], []
    for src in sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        fresh = (not force and not extra and os.path.exists(obj)
                 and os.path.getmtime(obj) > max(os.path.getmtime(src), newest_header))
        if not fresh:
            jobs.append((src, obj, extra or [], verbose))
    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        list(pool.map(_compile_one, jobs))
    cmd = [_nvcc(), *NVCC_FLAGS, "-shared", *objs, "-o", LIB_PATH]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return LIB_PATH


_TORCH_MARK = b"ffi-binding-torch="


def binding_torch() -> str | None:
    """The torch version ``_native.so`` was compiled against (None: there is no module)."""
    if not os.path.exists(BINDING_PATH):
        return None
    with open(BINDING_PATH, "rb") as f:
        after = f.read().partition(_TORCH_MARK)[2]
    return after.partition(b"\0")[0].decode("ascii", "replace")


def _binding_stale() -> bool:
    import torch

    if binding_torch() != torch.__version__:
        return True
    deps = [BINDING_SRC, os.path.join(INCLUDE, "ffi_b200.h")]
    return any(os.path.getmtime(d) > os.path.getmtime(BINDING_PATH) for d in deps)


def build_binding(force: bool = False, verbose: bool = False) -> str:
    """Compiles ``_native.so`` against the torch this interpreter imports and the CUDA library beside it."""
    if not force and not _binding_stale():
        return BINDING_PATH
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    build()
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include"), INCLUDE]
    libs = [p for p in cpp_extension.library_paths()]
    gxx = shutil.which("g++")
    if not gxx:
        raise CompilerMissing("g++ not found; the binding cannot be built")
    cmd = [gxx, "-std=c++17", "-O2", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DFFI_TORCH_VERSION="{torch.__version__}"', *(f"-isystem{i}" for i in includes),
           BINDING_SRC, "-o", BINDING_PATH, f"-L{PKG_DIR}", "-lffi_b200", "-Wl,-rpath,$ORIGIN",
           *(f"-L{p}" for p in libs), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return BINDING_PATH


if __name__ == "__main__":
    extra = ["-Xptxas", "-v"] if "--ptxas" in sys.argv else None
    print(build(force=True, verbose=True, extra=extra))
    print(build_binding(force=True, verbose=True))
