"""Calls of a kernel library's C entry points.

``EntryPoints(lib).leone_x(...)`` takes tensors (their data pointer is passed), ``None`` (a null pointer), ints (integers and
pointers) and floats (C floats), and returns the entry point's int.  The calls go through ``csrc/launch_call.cpp``, a CPython
extension built on first use: a call of 30 arguments takes 0.9 us there against 3.9 us through ctypes and the objects it wants.
Where the extension cannot be built (no Python headers, another platform) the same calls go through ctypes.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os

from ..csrc.build import BuildError, ensure_built

_BIND = None


def _through_ctypes(fn):
    def as_argument(a):
        if a is None:
            return None
        if isinstance(a, float):
            return ctypes.c_float(a)
        if isinstance(a, int):
            # As 64 bits whatever its size: an int without a type is a C int to ctypes, which writes four of the eight bytes of a place
            # on the stack, and the callee may read all eight (a stride, a stream).  One that reads an int takes the low half.
            if not -(1 << 63) <= a < 1 << 64:
                raise OverflowError("an argument does not fit 64 bits")
            return ctypes.c_longlong(a)
        return ctypes.c_void_p(a.data_ptr())

    return lambda *args: fn(*[as_argument(a) for a in args])


def _bind():
    """Makes a callable of a ctypes function."""
    global _BIND
    if _BIND is None:
        _BIND = _through_ctypes
        if os.environ.get("LEONE_NO_NATIVE_CALLS", "0") != "1":
            try:
                path = ensure_built("call")
                loader = importlib.machinery.ExtensionFileLoader("libleone_call", path)
                module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("libleone_call", path, loader=loader))
                loader.exec_module(module)
                _BIND = lambda fn: module.bind(ctypes.cast(fn, ctypes.c_void_p).value)      # noqa: E731
            except (BuildError, ImportError, OSError):
                pass
    return _BIND


class EntryPoints:
    def __init__(self, lib: ctypes.CDLL):
        self._lib = lib              # keeps the library loaded

    def __getattr__(self, name):
        if name.startswith("_"):
            raise AttributeError(name)
        entry = getattr(self._lib, name)
        if isinstance(self._lib, ctypes.CDLL):           # (a stand-in's entries are called as they are)
            entry = _bind()(entry)
        self.__dict__[name] = entry
        return entry
