"""
Loader of the autograd nodes in C++ (``csrc/pyext/autograd_nodes.cpp``): the same operators as the ``torch.autograd.Function`` classes of this
package, allocated and launched without the interpreter.

:func:`active` is None where the Python classes run: programs under ``torch.jit.trace`` (the tracer records a Python function as an operator of
its own and would record a C++ node as a constant), and installations without the extension.
"""

from __future__ import annotations
import importlib.util
import os
import torch
from . import _lib

_module = None
_tried = False


def _load():
    global _module, _tried
    with _lib._lock:
        if not _tried:
            path = os.path.join(_lib._LIB_DIR, "_autograd_nodes.so")
            if os.path.exists(path):
                spec = importlib.util.spec_from_file_location("_autograd_nodes", path)
                mod = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(mod)
                _module = mod
            _tried = True
    return _module


def active():
    """:return: the extension module, or None (see above). Callers have checked that the native kernels run (:func:`_lib.use_native`)"""
    mod = _module if _tried else _load()
    if mod is not None and torch._C._get_tracing_state() is None:
        return mod
    return None


def launches() -> int:
    """number of kernels that the nodes launched so far"""
    return _module.launches() if _module is not None else 0
