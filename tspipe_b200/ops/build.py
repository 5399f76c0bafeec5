"""Build and load ``libtspipe_b200.so`` (the sm_100a kernels under ``csrc/``).

The library is plain CUDA C with ``extern "C"`` launchers (no framework headers), compiled in-tree
with ``nvcc -gencode arch=compute_100a,code=sm_100a`` and loaded through ``ctypes``; tensors cross
the boundary as raw pointers plus the current CUDA stream handle.
"""
from __future__ import annotations

import ctypes
import hashlib
import os
import shutil
import subprocess
import threading
import warnings
from typing import List, Optional

_HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(os.path.dirname(_HERE))
CSRC = os.path.join(REPO, "csrc")
LIB_DIR = os.path.join(_HERE, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libtspipe_b200.so")
HASH_PATH = LIB_PATH + ".srchash"

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC"]

# Eager calls as C++ autograd functions (csrc/host): an extension module against the installed torch, next to the kernels
HOST_SOURCE = os.path.join(CSRC, "host", "eager.cpp")
HOST_NAME = "tspipe_eager"
HOST_PATH = os.path.join(LIB_DIR, HOST_NAME + ".so")

_lock = threading.Lock()
_lib: Optional[ctypes.CDLL] = None
_host = None
_no_host = False        # building or loading it has failed


def sources() -> List[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _source_hash() -> str:
    h = hashlib.sha256()
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, f), "rb") as fh:
                h.update(f.encode())
                h.update(fh.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def nvcc_path() -> Optional[str]:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else None


def is_fresh() -> bool:
    if not (os.path.exists(LIB_PATH) and os.path.exists(HASH_PATH)):
        return False
    with open(HASH_PATH) as f:
        return f.read().strip() == _source_hash()


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into one shared library (cross-compiles without a GPU)."""
    with _lock:
        if not force and is_fresh():
            return LIB_PATH
        nvcc = nvcc_path()
        if nvcc is None:
            raise RuntimeError("nvcc not found: cannot build the sm_100a kernels")
        os.makedirs(LIB_DIR, exist_ok=True)
        tmp = LIB_PATH + f".tmp{os.getpid()}"
        cmd = [nvcc] + NVCC_FLAGS + ["-I", CSRC, "-o", tmp] + sources() + ["-lcuda"]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed:\n{' '.join(cmd)}\n{res.stdout}\n{res.stderr}")
        if verbose:
            print(res.stderr)
        os.replace(tmp, LIB_PATH)
        with open(HASH_PATH, "w") as f:
            f.write(_source_hash())
        return LIB_PATH


def load() -> ctypes.CDLL:
    """Load the library, building it first when it is missing or stale.  Raises when neither a
    library nor a compiler is available - the CUDA ops never fall back silently."""
    global _lib
    if _lib is not None:
        return _lib
    if not is_fresh():
        if nvcc_path() is not None:
            build()
        elif not os.path.exists(LIB_PATH):
            raise RuntimeError(f"{LIB_PATH} is missing and nvcc is unavailable; run __graft_entry__.build()")
    with _lock:
        if _lib is None:
            _lib = ctypes.CDLL(LIB_PATH)
    return _lib


HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-DTORCH_EXTENSION_NAME={HOST_NAME}"]


def _host_command(out: str) -> List[str]:
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc_path() or "/usr/local/cuda/bin/nvcc"))
    incl = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
            sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++", *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[a for p in incl for a in ("-isystem", p)], HOST_SOURCE, "-o", out,
            "-L", LIB_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN",
            "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
            "-L", os.path.join(cuda, "lib64"), "-lcudart"]


def _host_hash() -> str:
    import sys

    import torch
    h = hashlib.sha256()
    for f in (HOST_SOURCE, os.path.join(CSRC, "tspipe_kernels.h")):
        with open(f, "rb") as fh:
            h.update(fh.read())
    h.update(f"{torch.__version__} {sys.version_info[:2]} {' '.join(HOST_FLAGS)}".encode())
    return h.hexdigest()


def host_is_fresh() -> bool:
    if not (os.path.exists(HOST_PATH) and os.path.exists(HOST_PATH + ".srchash")):
        return False
    with open(HOST_PATH + ".srchash") as f:
        return f.read().strip() == _host_hash()


def build_host() -> str:
    """Compile ``csrc/host/eager.cpp`` against the installed torch and the kernels' library."""
    build()
    with _lock:
        if host_is_fresh():
            return HOST_PATH
        tmp = HOST_PATH + f".tmp{os.getpid()}"
        cmd = _host_command(tmp)
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"g++ failed:\n{' '.join(cmd)}\n{res.stdout}\n{res.stderr}")
        os.replace(tmp, HOST_PATH)
        with open(HOST_PATH + ".srchash", "w") as f:
            f.write(_host_hash())
        return HOST_PATH


def load_host():
    """The extension module of the eager calls, built first when it is missing or stale; None where that cannot be done, with a
    warning the first time: their Python functions launch the same kernels, at a higher cost to the host.  A stale module is
    not loaded, since it is bound to the C++ interface of the torch that it was built against."""
    global _host, _no_host
    if _host is not None or _no_host:
        return _host
    load()
    try:
        if not host_is_fresh():
            if shutil.which("g++") is None:
                raise RuntimeError(f"{HOST_PATH} is missing or stale and g++ is unavailable")
            build_host()
        import importlib.util
        with _lock:
            if _host is None:
                spec = importlib.util.spec_from_file_location(HOST_NAME, HOST_PATH)
                module = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(module)
                _host = module
    except (RuntimeError, ImportError, OSError) as e:
        _no_host = True
        warnings.warn(f"eager calls stay with their Python functions: {e}", RuntimeWarning, stacklevel=2)
    return _host
