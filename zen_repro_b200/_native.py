"""Access to the in-tree native library (``_lib/libzen_b200.so``).

The library is plain CUDA with a C ABI: every entry point takes raw device
pointers, sizes and a ``cudaStream_t``.  ``lib()`` loads it once; on a machine
with a GPU a missing library is an error, never a silent fallback.
"""
from __future__ import annotations

import ctypes
import threading

import torch

from . import build as _build

_LOCK = threading.Lock()
_LIB = None


class NativeUnavailable(RuntimeError):
    pass


class _Library:
    """The library's functions as attributes, callable with ints (pointers included), floats, None and ctypes structures
    (csrc/fastcall.c)."""

    def __init__(self, path, fastcall):
        self._cdll, self._fast = ctypes.CDLL(str(path)), fastcall

    def __getattr__(self, name):
        addr = ctypes.cast(getattr(self._cdll, name), ctypes.c_void_p).value
        fn = self._fast.function(addr)
        self.__dict__[name] = fn
        return fn


def _load_fastcall(path):
    import importlib.machinery
    import importlib.util

    loader = importlib.machinery.ExtensionFileLoader("zen_fastcall", str(path))
    spec = importlib.util.spec_from_file_location("zen_fastcall", str(path), loader=loader)
    mod = importlib.util.module_from_spec(spec)
    loader.exec_module(mod)
    return mod


def lib() -> "_Library":
    """The loaded native library; built first where the ``.so`` is missing (needs nvcc) or the CPython extension beside it is
    missing or of another interpreter (needs a C compiler)."""
    global _LIB
    if _LIB is not None:
        return _LIB
    with _LOCK:
        if _LIB is None:
            path = _build.lib_path()
            if not path.exists() or not _build.fastcall_current():
                try:
                    path = _build.build() if not path.exists() else path
                    _build.build_fastcall()
                except Exception as e:  # pragma: no cover - depends on toolchain
                    raise NativeUnavailable(f"native library missing and build failed: {e}") from e
            _LIB = _Library(path, _load_fastcall(_build.fastcall_path()))
    return _LIB


def launch_count() -> int:
    """Kernels of this library launched so far in this process, as the library counts them where it launches them."""
    if _LIB is None:
        return 0
    n = ctypes.c_int64()
    _LIB.zen_launch_count(ctypes.byref(n))
    return n.value


def available() -> bool:
    """True when CUDA kernels can run here (a GPU is present and the library loads)."""
    if not torch.cuda.is_available():
        return False
    lib()
    return True


def stream_ptr(stream: torch.cuda.Stream | None = None) -> int:
    """The stream's handle; without an argument that of the current stream of the current device (through the raw getter:
    ``torch.cuda.current_stream`` builds a Stream object, 3.4 us a call)."""
    return stream.cuda_stream if stream is not None else torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def ptr(t: torch.Tensor | None) -> int:
    return 0 if t is None else t.data_ptr()


DTYPE_CODE = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise RuntimeError(f"{what} failed with CUDA/launcher code {rc}")
