"""Loader of lib/_fdma_torch.so, the native host path of the operators (csrc/fdma_torch.cpp): the checks, the route
choice, the allocations and the autograd node of a call in one C++ function instead of Python. Its functions return
None for calls they do not take (tracing, tensor subclasses, unusual layouts); the Python implementation then runs."""
import importlib.machinery
import importlib.util
import os

from . import _lib

_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "_fdma_torch.so")
_module = None


def load():
    """Loads the extension once. Raises RuntimeError when it has not been built."""
    global _module
    if _module is None:
        _lib.load()  # the C ABI library: raises when missing
        if not os.path.exists(_PATH):
            raise RuntimeError(f"{_PATH} not found: build it with `make -C flash-dmattn_b200/csrc`")
        loader = importlib.machinery.ExtensionFileLoader("_fdma_torch", _PATH)
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_fdma_torch", loader))
        loader.exec_module(module)
        module.init(_lib.LIB_PATH)
        _module = module
    return _module
