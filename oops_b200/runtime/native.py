"""Loader of the compiled host layer (``oops_b200/csrc/native.cpp``): argument checks of plain calls, autograd nodes,
allocation and launches.  Like the kernels it has no substitute: a missing module is an error."""

from __future__ import annotations

import importlib.machinery
import importlib.util

import torch  # noqa: F401  (its libraries must be loaded before the module that links to them)

from .._errors import OOpsUnsupportedError
from . import cabi

MODULE_PATH = cabi.LIB_PATH.parent / "_native.so"

_module = None


def native():
    """The module, loaded once."""
    global _module
    if _module is None:
        cabi.library()  # the kernels' library: present, and of the version this package expects
        if not MODULE_PATH.exists():
            raise RuntimeError(f"{MODULE_PATH} is missing: build it with `python -m oops_b200.csrc.build`")
        loader = importlib.machinery.ExtensionFileLoader("_native", str(MODULE_PATH))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_native", loader))
        loader.exec_module(module)
        module.set_unsupported_error(OOpsUnsupportedError)
        _module = module
    return _module


__all__ = ["MODULE_PATH", "native"]
