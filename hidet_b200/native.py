"""The plain case of every hot call, natively (csrc/host.cpp, built into lib/ under a name that carries the Python and torch
versions it was built against).

    out = native.linear(a, weight, scale, weight_layout, out, bias, residual, activation)

answers None for whatever is not the plain case; the caller then takes its general path.  The module is loaded with the
first call on a CUDA tensor, as the kernel library is.  Without a module for this Python and torch (or with one that does not
load) every function answers None, after one warning: the general paths are complete, only slower by some 10 us a call.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import sys
import warnings

import torch

from . import ffi

MODULE_NAME = 'hidet_b200_host'
LIB_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'lib')

# what csrc/host.cpp calls, in the order of its bind()
_BOUND = ('b200q_symmetric_quantize', 'b200q_symmetric_dequantize', 'b200q_embedding_dequantize', 'b200q_qlinear_workspace_bytes',
          'b200q_qlinear_f16_i8', 'b200q_qlinear_f16_i8_fused', 'b200q_qlinear_f16_u4_workspace_bytes', 'b200q_qlinear_f16_u4')
_FUNCTIONS = ('linear', 'quantize', 'dequantize', 'take', 'w4')
_module = None


def module_path() -> str:
    """Where the module for this Python and torch is: another torch has another name, so a stale one is never loaded."""
    return os.path.join(LIB_DIR, '{}.{}-torch-{}.so'.format(MODULE_NAME, sys.implementation.cache_tag, torch.__version__))


def _unavailable(*_):
    return None


def load():
    """The module, bound to the loaded kernel library, or None; its functions replace the stand-ins below."""
    global _module
    if _module is None:
        lib = ffi.load_library()
        path = module_path()
        try:
            loader = importlib.machinery.ExtensionFileLoader(MODULE_NAME, path)
            module = importlib.util.module_from_spec(importlib.util.spec_from_file_location(MODULE_NAME, path, loader=loader))
            loader.exec_module(module)
        except ImportError as e:
            warnings.warn('{} cannot be loaded ({}): calls take the Python path. Build it with `python -m hidet_b200.build`.'.format(path, e))
            for name in _FUNCTIONS:
                globals()[name] = _unavailable
            return None
        module.bind(*(ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _BOUND))
        _module = module
        for name in _FUNCTIONS:
            globals()[name] = getattr(module, name)
    return _module


def set_scratch(device: int, stream: int, address: int, nbytes: int) -> None:
    """Tells the module, if it is in use, which scratch a stream has (0 bytes: none)."""
    if _module is not None:
        _module.set_scratch(device, stream, address, nbytes)


def clear_scratch() -> None:
    if _module is not None:
        _module.clear_scratch()


def _stand_in(name):
    def first_call(x, *rest):
        if not (isinstance(x, torch.Tensor) and x.is_cuda):
            return None
        load()
        return globals()[name](x, *rest)

    return first_call


linear, quantize, dequantize, take, w4 = (_stand_in(name) for name in _FUNCTIONS)
