"""The compiled torch extension (``lib/_hcomm_torch.so``): the torch.distributed backend and the native calls."""
from __future__ import annotations

import ctypes
import importlib.util
import os
import sys
import threading
import warnings
from pathlib import Path

from . import _lib

_MODULE = None
_CALLS = False          # not looked for yet
_LOCK = threading.RLock()       # any thread's first call may be the one that loads
_PATH = Path(__file__).resolve().parent / "lib" / "_hcomm_torch.so"


def extension():
    """The extension module; built on first use when the shared object is missing."""
    global _MODULE
    if _MODULE is not None:
        return _MODULE
    import torch.distributed                      # noqa: F401  the backend class derives from one of its types
    with _LOCK:
        if _MODULE is None:
            _lib.load()                           # libhcomm.so first: the extension links against it
            if not _PATH.exists():
                from . import build
                build.build_torch_extension()
            spec = importlib.util.spec_from_file_location("_hcomm_torch", str(_PATH))
            mod = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(mod)
            sys.modules["_hcomm_torch"] = mod
            _MODULE = mod
    return _MODULE


def native_calls():
    """The extension where calls can take the short way through it, else None: without a GPU, with another build of the library
    selected, or where the extension was not built or does not load."""
    global _CALLS
    if _CALLS is not False:
        return _CALLS
    import torch
    with _LOCK:
        if _CALLS is False:
            found = failed = None
            if not os.environ.get("HCOMM_LIBRARY") and _PATH.exists() and torch.cuda.is_available():
                try:
                    found = extension()
                except ImportError as e:          # built against another torch
                    failed = e
            _CALLS = found
            if failed is not None:
                warnings.warn(f"{_PATH.name} does not load, calls take the longer way through Python: {failed}", stacklevel=2)
    return _CALLS


def entry(name: str) -> int:
    """Address of a C entry point in the loaded library."""
    return ctypes.cast(getattr(_lib.load(), name), ctypes.c_void_p).value


def _none(*_):
    return None


class Short:
    """One native call bound to its entry point.  Calling it gives None where the general way has to be taken."""

    __slots__ = ("_function", "_name", "_entry", "_call")

    def __init__(self, function: str, name: str):
        self._function, self._name, self._entry, self._call = function, name, 0, None

    def find(self):
        call = getattr(native_calls(), self._function, _none)
        self._entry = entry(self._name) if call is not _none else 0
        self._call = call
        return call

    def __call__(self, *args):
        call = self._call or self.find()
        r = call(self._entry, *args)
        if r.__class__ is int and r:
            _lib.check(r, self._name)
        return r
