"""Loads the native host path (csrc/host_fast.cpp, built into luma_b200/lib/ with the library) of the calls whose arguments are
exactly what an entry point takes, and hands it the C ABI's addresses from the ctypes handle in `ffi`.

Each function returns None, having done nothing, for anything it does not take; `high` and `low` then go
on in Python. An extension that was not built for this Python and this torch is not loaded: every call then takes the Python
path, with the same results and more host time, after one warning.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import warnings

import torch  # noqa: F401  (the extension links against the libraries that this import loads)

from . import build, error, ffi

PATH = build.host_path_file()


def _addresses():
    names = ([f"flash_attn_{s}" for s in ffi.DTYPE_SUFFIX] + [f"flash_attn_{s}_lse" for s in ffi.DTYPE_SUFFIX]
             + [f"flash_attn_varlen_{s}" for s in ffi.DTYPE_SUFFIX]
             + ["flash_attn_varlen_f16_total", "flash_attn_varlen_bf16_total"] + [f"flash_attn_with_kvcache_{s}" for s in ffi.DTYPE_SUFFIX]
             + ["flash_attn_kvcache_append"] + [f"luma_softmax_{s}" for s in ffi.DTYPE_SUFFIX] + ["flash_attn_last_error"])
    return tuple(ctypes.cast(getattr(ffi.lib, n), ctypes.c_void_p).value for n in names)


def _load():
    try:
        loader = importlib.machinery.ExtensionFileLoader("_host", str(PATH))
        native = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host", loader))
        loader.exec_module(native)
        native.bind(error.from_status, _addresses())
        return native
    except ImportError as e:
        warnings.warn(f"luma_b200: the native host path is not available ({e}); calls go through Python. "
                      "Build it with `python -m luma_b200.build`.", RuntimeWarning, stacklevel=2)
        return None


def _not_taken(*_):
    return None


_native = _load()

attn, low_attn, varlen, kvcache, append, softmax = (getattr(_native, name, _not_taken)
                                                    for name in ("attn", "low_attn", "varlen", "kvcache", "append", "softmax"))
