"""Loader and builder of the Flash-MVPA shared library (C ABI in ``include/mvpa.h``).

The library is compiled in-tree with ``nvcc`` for sm_100a only and bound through
``ctypes``; PyTorch supplies device memory and the CUDA stream, nothing else.
There is no fallback: if the library is missing and cannot be built, importing
callers get an ``ImportError``.
"""
from __future__ import annotations

import ctypes
import fcntl
import hashlib
import os
import shutil
import subprocess
import tempfile
import threading
from concurrent.futures import ThreadPoolExecutor
from contextlib import contextmanager, nullcontext

import torch
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

_HERE = os.path.dirname(os.path.abspath(__file__))
_CSRC = os.path.join(_HERE, "csrc")
_INCLUDE = os.path.join(os.path.dirname(_HERE), "include")
LIB_PATH = os.path.join(_HERE, "libmvpa_b200.so")
HASH_PATH = LIB_PATH + ".srchash"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]
FAST_MATH = "--use_fast_math"        # everywhere but in the files below, whose results are not rounded to 16 bits afterwards
PRECISE = ("mvpa_rows_f32.cu",)

MVPA_F32, MVPA_BF16, MVPA_F16 = 0, 1, 2

_lock = threading.Lock()
_lib = None


def sources():
    return sorted(os.path.join(_CSRC, f) for f in os.listdir(_CSRC) if f.endswith(".cu"))


def _source_hash() -> str:
    """Digest of everything the binary depends on (file times do not survive a copy)."""
    h = hashlib.sha256(" ".join([*NVCC_FLAGS, FAST_MATH, *PRECISE]).encode())
    deps = sorted(os.path.join(_CSRC, f) for f in os.listdir(_CSRC)) + [os.path.join(_INCLUDE, "mvpa.h")]
    for d in deps:
        h.update(os.path.basename(d).encode())
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _stale() -> bool:
    return is_stale(LIB_PATH, HASH_PATH, _source_hash)


def is_stale(lib_path, hash_path, digest) -> bool:
    if not (os.path.exists(lib_path) and os.path.exists(hash_path)):
        return True
    with open(hash_path) as f:
        return f.read().strip() != digest()


@contextmanager
def one_builder(lib_path):
    """Processes that start together on a fresh checkout build one after the other (and all but the first find it done).
    The lock is on the folder: nothing is left behind.  Where a file system has none, what `publish` does is still whole."""
    fd = os.open(os.path.dirname(lib_path), os.O_RDONLY)
    try:
        try:
            fcntl.flock(fd, fcntl.LOCK_EX)
        except OSError:
            pass
        yield
    finally:
        os.close(fd)


def publish(link, lib_path, hash_path, digest: str) -> None:
    """Put the library that `link(path)` writes, and then its digest, in place; nobody ever sees half of either."""
    with tempfile.TemporaryDirectory(dir=os.path.dirname(lib_path), prefix=".build") as place:
        new, new_hash = os.path.join(place, "lib"), os.path.join(place, "hash")
        link(new)
        with open(new_hash, "w") as f:
            f.write(digest)
        os.replace(new, lib_path)
        os.replace(new_hash, hash_path)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile ``csrc/*.cu`` into ``libmvpa_b200.so`` (cross-compiles without a GPU)."""
    if not force and not _stale():
        return LIB_PATH
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise ImportError("nvcc not found: cannot build libmvpa_b200.so")
    messages = []

    def run(args):
        res = subprocess.run([nvcc, *NVCC_FLAGS, *args], capture_output=True, text=True)
        if res.returncode != 0:
            raise ImportError("building libmvpa_b200.so failed:\n" + res.stdout + res.stderr)
        messages.append(res.stderr)

    def compile_one(src):
        obj = os.path.join(objects, os.path.basename(src) + ".o")
        fast = [] if os.path.basename(src) in PRECISE else [FAST_MATH]
        run([*fast, *(["-Xptxas=-v"] if verbose else []), "-I", _INCLUDE, "-I", _CSRC, "-c", src, "-o", obj])
        return obj

    try:
        with one_builder(LIB_PATH), tempfile.TemporaryDirectory() as objects, ThreadPoolExecutor() as pool:
            if force or _stale():
                digest = _source_hash()      # (of what is compiled, whatever happens to the sources meanwhile)
                publish(lambda path: run(["-shared", *pool.map(compile_one, sources()), "-o", path]), LIB_PATH, HASH_PATH, digest)
    except OSError as e:   # a folder that cannot be written to
        raise ImportError(f"building libmvpa_b200.so failed: {e}") from e
    if verbose:
        print("".join(messages))
    return LIB_PATH


class Problem(ctypes.Structure):
    _fields_ = [("B", ctypes.c_int32), ("H", ctypes.c_int32), ("Hkv", ctypes.c_int32),
                ("T", ctypes.c_int32), ("C", ctypes.c_int32), ("D", ctypes.c_int32),
                ("window", ctypes.c_int32), ("dtype", ctypes.c_int32),
                ("sm_scale", ctypes.c_float), ("flags", ctypes.c_int32),
                ("q_time_begin", ctypes.c_int32), ("q_time_count", ctypes.c_int32)]


class Tensor(ctypes.Structure):
    _fields_ = [("ptr", ctypes.c_void_p), ("stride_b", ctypes.c_int64),
                ("stride_h", ctypes.c_int64), ("stride_n", ctypes.c_int64)]


EXPORTS = ("mvpa_fwd", "mvpa_bwd", "mvpa_fwd_workspace_bytes", "mvpa_bwd_workspace_bytes",
           "mvpa_last_error_string", "mvpa_launch_count", "mvpa_abi_version",
           "mvpa_workspace_status", "mvpa_fwd_noalloc", "mvpa_bwd_status", "mvpa_noalloc_status",
           "mvpa_selftest_wait_timeout", "mvpa_rmsnorm", "mvpa_silu_mul", "mvpa_wave_encode_size",
           "mvpa_wave_encode", "mvpa_channel_mean", "mvpa_contrastive_logits", "mvpa_peer_gather", "mvpa_peer_signal",
           "mvpa_peer_wait", "mvpa_rmsnorm_bwd", "mvpa_rmsnorm_bwd_workspace_bytes", "mvpa_silu_mul_bwd")
ABI_VERSION = 3   # mvpa_abi_version() of the header this shim was written against


def lib() -> ctypes.CDLL:
    """The loaded library; builds it first when the sources are newer than the binary."""
    global _lib
    with _lock:
        if _lib is not None:
            return _lib
        if _stale():
            try:
                build()
            except ImportError:
                if not os.path.exists(LIB_PATH):
                    raise
        try:
            L = ctypes.CDLL(LIB_PATH)
        except OSError as e:  # no silent fallback: the CUDA library is the product
            raise ImportError(f"cannot load {LIB_PATH}: {e}") from e
        # a stale binary, kept because the rebuild failed: another version, or one from before an entry point was added
        version = L.mvpa_abi_version() if hasattr(L, "mvpa_abi_version") else None
        missing = [name for name in EXPORTS if not hasattr(L, name)]
        if version != ABI_VERSION or missing:
            raise ImportError(f"{LIB_PATH} has ABI version {version}, this shim needs {ABI_VERSION}"
                              + (f" with {', '.join(missing)}" if missing else "") + ": rebuild it (python __graft_entry__.py)")
        P, Tn, vp = ctypes.POINTER(Problem), ctypes.POINTER(Tensor), ctypes.c_void_p
        L.mvpa_fwd_workspace_bytes.restype = ctypes.c_size_t
        L.mvpa_fwd_workspace_bytes.argtypes = [P]
        L.mvpa_bwd_workspace_bytes.restype = ctypes.c_size_t
        L.mvpa_bwd_workspace_bytes.argtypes = [P]
        L.mvpa_fwd.restype = ctypes.c_int
        L.mvpa_fwd.argtypes = [P, Tn, Tn, Tn, vp, vp, vp, vp, vp, Tn, vp, vp, ctypes.c_size_t, vp]
        L.mvpa_bwd.restype = ctypes.c_int
        L.mvpa_bwd.argtypes = [P, Tn, Tn, Tn, vp, vp, vp, vp, vp, Tn, vp, Tn, Tn, Tn, Tn,
                               vp, vp, vp, vp, vp, vp, ctypes.c_size_t, vp]
        L.mvpa_fwd_noalloc.restype = ctypes.c_int
        L.mvpa_fwd_noalloc.argtypes = [P, Tn, Tn, Tn, vp, vp, vp, vp, vp, Tn, vp, vp]
        L.mvpa_workspace_status.restype = ctypes.c_int
        L.mvpa_workspace_status.argtypes = [vp, ctypes.c_size_t, vp]
        L.mvpa_bwd_status.restype = ctypes.c_int
        L.mvpa_bwd_status.argtypes = [P, vp, ctypes.c_size_t, vp]
        L.mvpa_noalloc_status.restype = ctypes.c_int
        L.mvpa_noalloc_status.argtypes = [vp]
        L.mvpa_selftest_wait_timeout.restype = ctypes.c_int
        L.mvpa_selftest_wait_timeout.argtypes = [vp, ctypes.c_size_t, ctypes.c_uint32, vp]
        i32, i64, f32 = ctypes.c_int32, ctypes.c_int64, ctypes.c_float
        L.mvpa_rmsnorm.restype = ctypes.c_int
        L.mvpa_rmsnorm.argtypes = [vp, vp, vp, vp, vp, i64, i32, f32, i32, vp]
        L.mvpa_silu_mul.restype = ctypes.c_int
        L.mvpa_silu_mul.argtypes = [vp, vp, i64, vp, i64, i64, i32, i32, vp]
        L.mvpa_rmsnorm_bwd_workspace_bytes.restype = ctypes.c_size_t
        L.mvpa_rmsnorm_bwd_workspace_bytes.argtypes = [i64, i32]
        L.mvpa_rmsnorm_bwd.restype = ctypes.c_int
        L.mvpa_rmsnorm_bwd.argtypes = [vp, vp, vp, vp, vp, vp, i64, i32, f32, i32, vp, ctypes.c_size_t, vp]
        L.mvpa_silu_mul_bwd.restype = ctypes.c_int
        L.mvpa_silu_mul_bwd.argtypes = [vp, vp, i64, vp, i64, vp, vp, i64, i64, i32, i32, vp]
        L.mvpa_wave_encode_size.restype = i32
        L.mvpa_wave_encode_size.argtypes = [i32, ctypes.POINTER(i32), i32]
        L.mvpa_wave_encode.restype = ctypes.c_int
        L.mvpa_wave_encode.argtypes = [vp, i64, i32, ctypes.POINTER(f32), ctypes.POINTER(f32), vp, vp, i64, i32, i64,
                                       i32, f32, vp]
        L.mvpa_peer_signal.restype = ctypes.c_int
        L.mvpa_peer_signal.argtypes = [vp, i32, ctypes.c_uint32, vp, vp]
        L.mvpa_peer_wait.restype = ctypes.c_int
        L.mvpa_peer_wait.argtypes = [vp, i32, ctypes.c_uint32, vp, ctypes.c_uint32, vp, vp]
        L.mvpa_peer_gather.restype = ctypes.c_int
        L.mvpa_peer_gather.argtypes = [vp, vp, vp, i32, vp]
        L.mvpa_channel_mean.restype = ctypes.c_int
        L.mvpa_channel_mean.argtypes = [vp, vp, i32, i32, i32, i32, i32, vp]
        L.mvpa_contrastive_logits.restype = ctypes.c_int
        L.mvpa_contrastive_logits.argtypes = [vp, vp, vp, vp, i32, i32, i32, i32, i32, f32, i32, vp]
        L.mvpa_last_error_string.restype = ctypes.c_char_p
        L.mvpa_launch_count.restype = ctypes.c_uint64
        _lib = L
        return L


_SAME_DEVICE = nullcontext()


def on_device(device):
    """Context in which `device` is the current CUDA device; costs nothing when it already is."""
    return _SAME_DEVICE if device.index == torch.cuda.current_device() else torch.cuda.device(device)


def untraced() -> bool:
    """No forward-mode level, functorch transform, tracer, compiler or mode that sees each operation is watching the
    current call.  (A default device is a function mode as well; it only fills in where new tensors live.)"""
    return (torch.autograd.forward_ad._current_level < 0 and torch._C._functorch.peek_interpreter_stack() is None
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling() and not torch._C._len_torch_dispatch_stack()
            and (not torch._C._len_torch_function_stack()
                 or all(isinstance(m, DeviceContext) for m in _get_current_function_mode_stack())))


def last_error() -> str:
    return lib().mvpa_last_error_string().decode()


def check(status: int, what: str) -> None:
    """Raise like the reference does (`attentions/attn.py:1034-1045`): RuntimeError."""
    if status != 0:
        raise RuntimeError(f"{what} failed (status {status}): {last_error()}")
