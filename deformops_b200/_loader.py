"""Loads ``libmsda_b200.so`` (the C ABI of ``include/msda_b200.h``) through ctypes.

Plays the role of the reference's kernel-library loader
(``lazy_extension`` / ``define_library``, ``sources/deformops/core/build.py:75-137``
and ``:1116-1296``) reduced to what this build needs: one local library, loaded once
per process under a lock, a failed load is not memoised, and a forked child gets a fresh
lock.  There is no CPU path behind it: if the library cannot be loaded the call fails
with :class:`KernelUnavailableError`.
"""

from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import threading
import warnings

from ._build import (LIB_PATH, build_host_module, build_library, host_module_path, is_stale)
from .core.errors import KernelBuildError, KernelUnavailableError

__all__ = ["ABI_VERSION", "Shim", "host_module", "library_path", "load_library", "loaded"]

ABI_VERSION = 5

_lock = threading.Lock()
_shim: "Shim | None" = None
_host = None
_host_tried = False


def _reset_lock_in_child() -> None:
    global _lock
    _lock = threading.Lock()


os.register_at_fork(after_in_child=_reset_lock_in_child)

_i64, _vp, _int = ctypes.c_int64, ctypes.c_void_p, ctypes.c_int


class Shim:
    """Typed handles on the exported functions of the library."""

    #: every symbol ``include/msda_b200.h`` declares
    SYMBOLS = ("msda_b200_abi_version", "msda_b200_last_error", "msda_b200_launches", "msda_b200_forward",
               "msda_b200_backward", "msda_b200_backward_scratch_bytes",
               "msda_b200_backward_workspace_bytes", "msda_b200_backward_offsets_workspace_bytes",
               "msda_b200_column_sums",
               "msda_b200_column_sums_scratch_bytes",
               "msda_b200_forward_offsets", "msda_b200_backward_offsets",
               "msda_b200_backward_static_scratch", "msda_b200_launch_geometry")

    def __init__(self, path: str):
        self.path = path
        self.lib = ctypes.CDLL(path)
        missing = [s for s in self.SYMBOLS if not hasattr(self.lib, s)]
        if missing:
            raise KernelUnavailableError(f"{path} does not export {missing}")
        self.lib.msda_b200_abi_version.restype = _int
        self.lib.msda_b200_abi_version.argtypes = []
        self.lib.msda_b200_last_error.restype = ctypes.c_char_p
        self.lib.msda_b200_last_error.argtypes = []
        self.lib.msda_b200_launches.restype = None
        self.lib.msda_b200_launches.argtypes = [ctypes.POINTER(_i64), ctypes.POINTER(_i64)]
        self.forward = self.lib.msda_b200_forward
        self.forward.restype = _int
        self.forward.argtypes = [_vp] * 6 + [_i64] * 7 + [_int, _int, _int, _vp]
        self.backward = self.lib.msda_b200_backward
        self.backward.restype = _int
        self.backward.argtypes = ([_vp] * 10 + [_i64, _i64] + [_i64] * 7
                                  + [_int, _int, _int, _int, _vp])
        self.scratch_bytes = self.lib.msda_b200_backward_scratch_bytes
        self.scratch_bytes.restype = _i64
        self.scratch_bytes.argtypes = [_i64] * 7 + [_int]
        self.workspace_bytes = self.lib.msda_b200_backward_workspace_bytes
        self.workspace_bytes.restype = _i64
        self.workspace_bytes.argtypes = [_i64] * 7 + [_int, _int]
        self.offsets_workspace_bytes = self.lib.msda_b200_backward_offsets_workspace_bytes
        self.offsets_workspace_bytes.restype = _i64
        self.offsets_workspace_bytes.argtypes = [_i64] * 7 + [_int, _int]
        self.column_sums = self.lib.msda_b200_column_sums
        self.column_sums.restype = _int
        self.column_sums.argtypes = [_vp, _vp, _vp, _i64, _i64, _int, _vp]
        self.column_sums_scratch_bytes = self.lib.msda_b200_column_sums_scratch_bytes
        self.column_sums_scratch_bytes.restype = _i64
        self.column_sums_scratch_bytes.argtypes = [_i64, _i64]
        self.forward_offsets = self.lib.msda_b200_forward_offsets
        self.forward_offsets.restype = _int
        self.forward_offsets.argtypes = ([_vp] * 4 + [_int, _vp, _int, _vp, _vp] + [_i64] * 7
                                         + [_int, _int, _int, _vp])
        self.backward_offsets = self.lib.msda_b200_backward_offsets
        self.backward_offsets.restype = _int
        self.backward_offsets.argtypes = ([_vp] * 4 + [_int, _vp, _int] + [_vp] * 6
                                          + [_i64, _i64] + [_i64] * 7
                                          + [_int, _int, _int, _int, _vp])
        self.backward_static_scratch = self.lib.msda_b200_backward_static_scratch
        self.backward_static_scratch.restype = _int
        self.backward_static_scratch.argtypes = ([_vp] * 9 + [_i64] + [_i64] * 7
                                                 + [_int, _int, _int, _vp])
        self.launch_geometry = self.lib.msda_b200_launch_geometry
        self.launch_geometry.restype = _int
        self.launch_geometry.argtypes = [_i64] * 6 + [_int, _int, ctypes.POINTER(_i64),
                                         ctypes.POINTER(_int), ctypes.POINTER(_i64),
                                         ctypes.POINTER(_i64)]
        got = self.lib.msda_b200_abi_version()
        if got != ABI_VERSION:
            raise KernelUnavailableError(
                f"{path} has ABI version {got}, this package needs {ABI_VERSION}: rebuild it")

    def launches(self) -> "tuple[int, int]":
        """Kernels and memsets the library has enqueued since it was loaded."""
        kernels, memsets = _i64(), _i64()
        self.lib.msda_b200_launches(ctypes.byref(kernels), ctypes.byref(memsets))
        return kernels.value, memsets.value

    def last_error(self) -> str:
        return self.lib.msda_b200_last_error().decode("utf-8", "replace")


def library_path() -> str:
    return os.environ.get("DEFORMOPS_B200_LIBRARY", str(LIB_PATH))


def loaded() -> bool:
    return _shim is not None


def load_library(*, compile: "bool | None" = None) -> Shim:
    """Load the kernel library once per process and return its :class:`Shim`.

    ``compile`` (default: environment ``DEFORMOPS_B200_COMPILE``, on unless it is ``0``)
    allows building the library with ``nvcc`` when it is missing or older than its sources.
    """
    global _shim
    if _shim is not None:
        return _shim
    with _lock:
        if _shim is not None:
            return _shim
        path = library_path()
        if compile is None:
            compile = os.environ.get("DEFORMOPS_B200_COMPILE", "1") != "0"
        if path == str(LIB_PATH) and compile and is_stale():
            try:
                build_library()
            except Exception as exc:  # noqa: BLE001 - surfaced as a typed error
                if not LIB_PATH.exists():
                    raise KernelBuildError(f"cannot build {LIB_PATH}: {exc}") from exc
        if not os.path.exists(path):
            raise KernelUnavailableError(
                f"kernel library {path} is missing; build it with "
                "`python -m deformops_b200._build` (needs nvcc). There is no CPU path.")
        try:
            _shim = Shim(path)
        except OSError as exc:
            raise KernelUnavailableError(f"cannot load {path}: {exc}") from exc
        return _shim


def host_module():
    """The native eager call path (``csrc/torch_host.cpp``) bound to the loaded library, or
    ``None`` where it cannot be had: the Python operators serve every call then, slower.

    Built on first use like the library itself, unless ``DEFORMOPS_B200_COMPILE=0``.
    """
    global _host, _host_tried
    if _host_tried:
        return _host
    shim = load_library()
    with _lock:
        if _host_tried:
            return _host
        try:
            path = host_module_path()
            if os.environ.get("DEFORMOPS_B200_COMPILE", "1") != "0":
                path = build_host_module()
            loader = importlib.machinery.ExtensionFileLoader("msda_b200_host", str(path))
            spec = importlib.util.spec_from_file_location("msda_b200_host", path, loader=loader)
            module = importlib.util.module_from_spec(spec)
            loader.exec_module(module)
            functions = (shim.forward, shim.backward, shim.forward_offsets, shim.backward_offsets,
                         shim.workspace_bytes, shim.lib.msda_b200_last_error,
                         shim.lib.msda_b200_column_sums,
                         shim.lib.msda_b200_column_sums_scratch_bytes,
                         shim.offsets_workspace_bytes)
            module.bind(*(ctypes.cast(f, ctypes.c_void_p).value for f in functions))
            _host = module
        except Exception as exc:  # noqa: BLE001 - the Python operators remain
            warnings.warn(f"deformops_b200: the native call path is not available ({exc}); "
                          "calls go through the Python operators", RuntimeWarning, stacklevel=3)
        _host_tried = True
        return _host
