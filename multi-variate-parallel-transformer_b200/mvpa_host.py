"""Loader and builder of the host extension (``csrc_host/mvpa_host.cpp``): the operator's and the block's calls around the C
ABI of the CUDA library, as single native calls on torch tensors.

Compiled in-tree with the host compiler against the installed torch, like the CUDA library is with nvcc; the digest of
what it was built from (its source, the C header, the versions of torch and Python) stands beside it.
"""
from __future__ import annotations

import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import threading
import warnings

import torch
from torch.utils._device import DeviceContext

import mvpa_native as _nat

_HERE = os.path.dirname(os.path.abspath(__file__))
_SOURCE = os.path.join(_HERE, "csrc_host", "mvpa_host.cpp")
_HEADER = os.path.join(os.path.dirname(_HERE), "include", "mvpa.h")
_NAME = "mvpa_host_b200"
LIB_PATH = os.path.join(_HERE, _NAME + ".so")
HASH_PATH = LIB_PATH + ".srchash"
FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-DNDEBUG", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
LIBS = ["c10", "c10_cuda", "torch_cpu", "torch_cuda", "torch_python"]

_lock = threading.Lock()
_module = None
_refused = False      # the extension cannot be built or loaded here


def _source_hash() -> str:
    h = hashlib.sha256(" ".join([*FLAGS, *LIBS, torch.__version__, sys.version]).encode())
    for path in (_SOURCE, _HEADER):
        with open(path, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _stale() -> bool:
    return _nat.is_stale(LIB_PATH, HASH_PATH, _source_hash)


def build(force: bool = False) -> str:
    """Compile the extension (needs no GPU)."""
    if not force and not _stale():
        return LIB_PATH
    compiler = os.environ.get("CXX") or shutil.which("g++") or "g++"
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    includes = [os.path.dirname(_HEADER), sysconfig.get_paths()["include"], os.path.join(root, "include"),
                os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]

    def link(path):
        res = subprocess.run([compiler, *FLAGS, *(f"-I{i}" for i in includes), _SOURCE, f"-L{os.path.join(root, 'lib')}",
                              *(f"-l{name}" for name in LIBS), "-o", path], capture_output=True, text=True)
        if res.returncode != 0:
            raise ImportError(f"building {_NAME}.so failed:\n" + res.stdout + res.stderr)

    try:
        with _nat.one_builder(LIB_PATH):
            if force or _stale():
                _nat.publish(link, LIB_PATH, HASH_PATH, _source_hash())
    except OSError as e:   # no compiler, or a folder that cannot be written to
        raise ImportError(f"building {_NAME}.so failed: {e}") from e
    return LIB_PATH


def module():
    """The loaded extension; builds it first when its sources are newer than the binary.  (A binary built for another torch is
    refused.)"""
    global _module
    if _module is None:
        with _lock:
            if _module is None:
                build()
                _nat.lib()
                loader = importlib.machinery.ExtensionFileLoader(_NAME, LIB_PATH)
                loaded = importlib.util.module_from_spec(importlib.util.spec_from_file_location(_NAME, LIB_PATH, loader=loader))
                loader.exec_module(loaded)
                loaded.init(_nat.LIB_PATH, DeviceContext)
                _module = loaded
    return _module


def available() -> bool:
    """Whether there is an extension.  A box without a C++ compiler or torch's headers can use a CUDA library that came ready
    built: the Python paths around the same kernels serve it, with a warning."""
    global _refused
    if _module is None and not _refused:
        _nat.lib()                      # (without the CUDA library nothing works: that error is its own)
        try:
            module()
        except ImportError as e:
            _refused = True
            warnings.warn(f"{e}\nCalls go through Python instead: the same kernels and results, more host time.", RuntimeWarning)
    return _module is not None


def usable(t) -> bool:
    """Whether a call on `t` may go to the extension at all: an ordinary CUDA tensor, no compiler looking on, no forward-mode
    level.  (The extension itself sees modes, transforms, tracers and every tensor's layout.)"""
    return ((type(t) is torch.Tensor or type(t) is torch.nn.Parameter) and not torch.compiler.is_compiling()
            and torch.autograd.forward_ad._current_level < 0 and t.is_cuda and (_module is not None or available()))
