"""Loads luma_b200/lib/_host.so (csrc/host_fast.cpp), the native host path of the calls whose arguments are exactly
what an entry point takes, and hands it the C ABI's addresses from the ctypes handle in `ffi`.

Each function returns None, having done nothing, for anything it does not take; `high` and `low` then go
on in Python. The extension is built with the library (luma_b200/build.py); a missing one is an ImportError.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
from pathlib import Path

import torch  # noqa: F401  (the extension links against the libraries that this import loads)

from . import error, ffi

PATH = Path(__file__).resolve().parent / "lib" / "_host.so"

if not PATH.exists():
    raise ImportError(f"{PATH} is missing: build it with `python -m luma_b200.build`")

_loader = importlib.machinery.ExtensionFileLoader("_host", str(PATH))
_native = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host", _loader))
_loader.exec_module(_native)


def _addresses():
    names = ([f"flash_attn_{s}" for s in ffi.DTYPE_SUFFIX] + [f"flash_attn_{s}_lse" for s in ffi.DTYPE_SUFFIX]
             + [f"flash_attn_varlen_{s}" for s in ffi.DTYPE_SUFFIX]
             + ["flash_attn_varlen_f16_total", "flash_attn_varlen_bf16_total"] + [f"flash_attn_with_kvcache_{s}" for s in ffi.DTYPE_SUFFIX]
             + ["flash_attn_kvcache_append"] + [f"luma_softmax_{s}" for s in ffi.DTYPE_SUFFIX] + ["flash_attn_last_error"])
    return tuple(ctypes.cast(getattr(ffi.lib, n), ctypes.c_void_p).value for n in names)


_native.bind(error.from_status, _addresses())

attn = _native.attn
low_attn = _native.low_attn
varlen = _native.varlen
kvcache = _native.kvcache
append = _native.append
softmax = _native.softmax
