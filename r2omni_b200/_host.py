"""The native host module (``csrc/host_ext.cpp``): tensor checks, cache allocation and launches without Python or ctypes
in between."""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os

from . import _lib
from .build import HOST_LIB

_module = None


def host():
    """The loaded module.  There is no fallback: a missing module is an error."""
    global _module
    if _module is None:
        if not os.path.exists(HOST_LIB):
            raise RuntimeError(f"{HOST_LIB} is missing: build it with `python -m r2omni_b200.build`")
        _lib.lib()   # the C ABI library it links against
        loader = importlib.machinery.ExtensionFileLoader("_r2k_host", HOST_LIB)
        spec = importlib.util.spec_from_file_location("_r2k_host", HOST_LIB, loader=loader)
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
        _module = module
    return _module
