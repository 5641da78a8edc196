"""Loads the native host path (``csrc/torch_ext.cpp``) and binds it to the C-ABI library.

As with the library itself there is no fallback: if the extension is missing, the first call on CUDA
tensors fails with instructions to build it.
"""

from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import threading

from . import _cabi
from ._paths import EXT_NAME, EXT_PATH

_ext = None
_lock = threading.Lock()


def loaded():
    """The extension module if it has been loaded, else None."""
    return _ext


def load(accurate_override: int = -1):
    """Load (once) and bind the extension; `accurate_override` is the state of ``accurate_sigmoid()``."""
    global _ext
    if _ext is not None:
        return _ext
    with _lock:
        if _ext is not None:
            return _ext
        if not os.path.exists(EXT_PATH):
            raise ImportError(
                f"{EXT_PATH} is missing: build it with `python -m triton_sigmoid_b200.build` "
                "(needs nvcc with sm_100a support and g++). This package has no other execution path."
            )
        lib = _cabi.load()
        loader = importlib.machinery.ExtensionFileLoader(EXT_NAME, EXT_PATH)
        mod = importlib.util.module_from_spec(importlib.util.spec_from_loader(EXT_NAME, loader))
        loader.exec_module(mod)
        addr = lambda fn: ctypes.cast(fn, ctypes.c_void_p).value  # noqa: E731
        mod.bind(addr(lib.sigattn_fwd), addr(lib.sigattn_bwd), addr(lib.sigattn_last_error), addr(lib.sigattn_device_status))
        mod.set_accurate(accurate_override)
        _ext = mod
    return _ext
