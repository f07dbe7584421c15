"""The package's host module (csrc/host.cpp): whole eager calls -- checks, allocation, launches -- in native code."""
from __future__ import annotations

import importlib.machinery
import importlib.util

from . import _abi

MODULE = _abi.LIBRARY.with_name("inkling_b200_host.so")
_module = None


def host():
    global _module
    if _module is None:
        _abi.lib()   # the CUDA library first: the module links against it
        if not MODULE.exists():
            raise RuntimeError(f"{MODULE} is missing: build it with `python {MODULE.parent / 'csrc' / 'build.py'}`. "
                               "There is no Python fallback for the calls it serves.")
        loader = importlib.machinery.ExtensionFileLoader("inkling_b200_host", str(MODULE))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("inkling_b200_host", loader))
        loader.exec_module(module)
        _module = module
    return _module
