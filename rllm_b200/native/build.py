"""Compiles ``native/csrc/<name>.cc`` with g++ into ``_build/<name>.<hash>.so``
next to the sources (or under the system's temporary folder if the package
folder cannot be written) the first time it is asked for, and loads it with
ctypes, or as an extension module where it is one.  The hash covers the source
and the flags (for an extension the versions of Python and PyTorch too, whose
headers it includes), so an edited source is rebuilt and a stale library is
never loaded.
"""
from __future__ import annotations

import ctypes
import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import threading
from typing import Dict, List

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
CXX_FLAGS = ["-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-Wall"]
SOURCES = ["cache_core"]
EXTENSIONS = ["launch"]           # modules of the interpreter

_lock = threading.Lock()
_loaded: Dict[str, ctypes.CDLL] = {}


class NativeBuildError(RuntimeError):
    pass


def _compiler() -> str:
    for cand in (os.environ.get("CXX"), shutil.which("g++"), shutil.which("c++"), shutil.which("clang++")):
        if cand and (os.path.isfile(cand) or shutil.which(cand)):
            return cand
    raise NativeBuildError("no C++ compiler found (set CXX); the engine's cache manager is C++")


def _build_dir() -> str:
    d = os.path.join(_HERE, "_build")
    try:
        os.makedirs(d, exist_ok=True)
        probe = os.path.join(d, f".probe{os.getpid()}")
        with open(probe, "w"):
            pass
        os.remove(probe)
        return d
    except OSError:
        d = os.path.join(tempfile.gettempdir(), f"rllm_b200_native_{os.getuid()}")
        os.makedirs(d, exist_ok=True)
        return d


def _flags(name: str) -> List[str]:
    if name not in EXTENSIONS:
        return CXX_FLAGS
    import torch

    from ..kernels import build as kernels_build
    top = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(kernels_build.find_nvcc()))), "include")
    includes = [sysconfig.get_paths()["include"], os.path.join(top, "include"),
                os.path.join(top, "include", "torch", "csrc", "api", "include"), cuda]
    return CXX_FLAGS + [f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + \
        [a for d in includes for a in ("-isystem", d)]


def _libraries(name: str) -> List[str]:
    """What an extension is linked with: PyTorch's own libraries, which are loaded when it is."""
    if name not in EXTENSIONS:
        return []
    import torch
    return ["-L" + os.path.join(os.path.dirname(torch.__file__), "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"]


def library_path(name: str) -> str:
    h = hashlib.sha256(" ".join(CXX_FLAGS).encode())
    if name in EXTENSIONS:
        import torch
        h.update(f"{sys.version} {torch.__version__}".encode())
    with open(os.path.join(CSRC, name + ".cc"), "rb") as f:
        h.update(f.read())
    return os.path.join(_build_dir(), f"{name}.{h.hexdigest()[:16]}.so")


def compile_library(name: str, verbose: bool = True) -> str:
    src = os.path.join(CSRC, name + ".cc")
    if not os.path.isfile(src):
        raise NativeBuildError(f"no source {src}")
    out = library_path(name)
    if os.path.isfile(out):
        return out
    tmp = f"{out}.{os.getpid()}.tmp"
    cmd = [_compiler()] + _flags(name) + ["-o", tmp, src] + _libraries(name)
    if verbose:
        print(f"[rllm_b200] compiling {name}.cc ...", file=sys.stderr, flush=True)
    proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if proc.returncode != 0:
        try:
            os.remove(tmp)
        except OSError:
            pass
        raise NativeBuildError(f"{cmd[0]} failed on {name}.cc:\n{proc.stdout}")
    os.replace(tmp, out)
    for fn in os.listdir(os.path.dirname(out)):        # libraries of older versions of this source
        if fn.startswith(name + ".") and fn.endswith(".so") and os.path.join(os.path.dirname(out), fn) != out:
            try:
                os.remove(os.path.join(os.path.dirname(out), fn))
            except OSError:
                pass
    return out


def load_library(name: str) -> ctypes.CDLL:
    with _lock:
        lib = _loaded.get(name)
        if lib is None:
            lib = _loaded[name] = ctypes.CDLL(compile_library(name))
        return lib


_modules: Dict[str, object] = {}


def load_extension(name: str):
    with _lock:
        module = _modules.get(name)
        if module is None:
            import torch  # noqa: F401  (its libraries, which the extension needs)
            loader = importlib.machinery.ExtensionFileLoader(name, compile_library(name))
            module = importlib.util.module_from_spec(importlib.util.spec_from_loader(name, loader))
            loader.exec_module(module)
            _modules[name] = module
        return module


def build_all(verbose: bool = True):
    return [compile_library(n, verbose) for n in SOURCES + EXTENSIONS]
