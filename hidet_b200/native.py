"""The plain case of every hot call, natively (csrc/host.cpp, built into lib/hidet_b200_host.so).

    out = native.linear(a, weight, scale, weight_layout, out, bias, residual, activation)

answers None for whatever is not the plain case; the caller then takes its general path.  The module is loaded with the
first call on a CUDA tensor, as the kernel library is; a missing module raises like a missing kernel library.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os

import torch

from . import ffi

MODULE_NAME = 'hidet_b200_host'
MODULE_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'lib', MODULE_NAME + '.so')

# what csrc/host.cpp calls, in the order of its bind()
_BOUND = ('b200q_symmetric_quantize', 'b200q_symmetric_dequantize', 'b200q_embedding_dequantize', 'b200q_qlinear_workspace_bytes',
          'b200q_qlinear_f16_i8', 'b200q_qlinear_f16_i8_fused', 'b200q_qlinear_f16_u4_workspace_bytes', 'b200q_qlinear_f16_u4')
_FUNCTIONS = ('linear', 'quantize', 'dequantize', 'take', 'w4')
_module = None


def load():
    """The module, bound to the loaded kernel library; its functions replace the stand-ins below."""
    global _module
    if _module is None:
        lib = ffi.load_library()
        if not os.path.exists(MODULE_PATH):
            raise ffi.BackendException('{} not found. Build it with `python -m hidet_b200.build`.'.format(MODULE_PATH))
        loader = importlib.machinery.ExtensionFileLoader(MODULE_NAME, MODULE_PATH)
        spec = importlib.util.spec_from_file_location(MODULE_NAME, MODULE_PATH, loader=loader)
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
        module.bind(*(ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _BOUND))
        _module = module
        for name in _FUNCTIONS:
            globals()[name] = getattr(module, name)
    return _module


def _stand_in(name):
    def first_call(x, *rest):
        if not (isinstance(x, torch.Tensor) and x.is_cuda):
            return None
        return getattr(load(), name)(x, *rest)

    return first_call


linear, quantize, dequantize, take, w4 = (_stand_in(name) for name in _FUNCTIONS)
