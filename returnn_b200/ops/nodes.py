"""
Loader of the autograd nodes in C++ (``csrc/pyext/autograd_nodes.cpp``): the same operators as the ``torch.autograd.Function`` classes of this
package, allocated and launched without the interpreter.

:func:`active` is None where the Python classes run: programs under ``torch.jit.trace`` (the tracer records a Python function as an operator of
its own and would record a C++ node as a constant), and installations without an extension that fits. The extension is compiled against one
version of torch and of Python, which its file name carries: another one's is not loaded. Where there is only such a one, or where it cannot
be loaded, the Python classes take its place after a warning (the kernels are those of ``librb200.so`` either way).
"""

from __future__ import annotations
import glob
import importlib.util
import os
import re
import sys
import warnings
import torch
from . import _lib

_module = None
_tried = False
_STEM = "_autograd_nodes"


def file_name() -> str:
    """name of the extension for the running torch and Python"""
    return re.sub(r"[^\w.-]", "_", "%s-torch%s-%s" % (_STEM, torch.__version__, sys.implementation.cache_tag)) + ".so"


def _load():
    global _module, _tried
    with _lib._lock:
        if not _tried:
            path, why = os.path.join(_lib._LIB_DIR, file_name()), None
            if os.path.exists(path):
                try:
                    spec = importlib.util.spec_from_file_location(_STEM, path)
                    mod = importlib.util.module_from_spec(spec)
                    spec.loader.exec_module(mod)
                    _module = mod
                except (ImportError, OSError) as exc:
                    why = "%s cannot be loaded (%s)" % (path, exc)
            else:
                other = glob.glob(os.path.join(glob.escape(_lib._LIB_DIR), _STEM + "*.so"))
                if other:
                    why = "%s is not there, only %s" % (path, ", ".join(os.path.basename(f) for f in sorted(other)))
            _tried = True
            if why:
                warnings.warn("Autograd nodes: %s. The Python functions run in their place, with more time on the host. "
                              "Build: python -m returnn_b200.ops.build" % why, RuntimeWarning, stacklevel=3)
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
