"""The native host path without a GPU: found by the versions it was built for, done without where it is missing."""
import os

import pytest
import torch

from hidet_b200 import build, native
from hidet_b200.runtime import workspaces


@pytest.fixture
def fresh(monkeypatch):
    """native as it is before its first call"""
    monkeypatch.setattr(native, '_module', None)
    for name in native._FUNCTIONS:
        monkeypatch.setattr(native, name, native._stand_in(name))
    return monkeypatch


def test_built_module_answers_none_for_cpu_tensors(fresh):
    module = native.load()
    assert module is not None and native.linear is module.linear
    a, wq, scale = torch.zeros(1, 16).half(), torch.zeros(16, 16, dtype=torch.int8), torch.zeros(16).half()
    assert native.linear(a, wq, scale, 'KN', None, None, None, None) is None
    assert native.quantize(a, 'int8', 0) is None and native.dequantize(wq, scale, 0) is None
    assert native.take(wq, scale, torch.zeros(3, dtype=torch.int64)) is None and native.w4(a, wq, scale, None, 16, 16, 16) is None


def test_another_torch_has_another_module(fresh):
    path = native.module_path()
    fresh.setattr(torch, '__version__', '0.0.1')
    assert native.module_path() != path and not os.path.exists(native.module_path())


def test_missing_or_broken_module_is_done_without(fresh, tmp_path):
    fresh.setattr(native, 'LIB_DIR', str(tmp_path))
    with pytest.warns(UserWarning, match='cannot be loaded'):
        assert native.load() is None
    assert all(getattr(native, name)(1, 2, 3) is None for name in native._FUNCTIONS)
    open(native.module_path(), 'w').write('not a library')
    with pytest.warns(UserWarning, match='cannot be loaded'):
        assert native.load() is None
    native.set_scratch(0, 0, 0, 0)
    workspaces.clear()


def test_kernel_library_builds_without_a_host_compiler(fresh, tmp_path):
    fresh.setattr(native, 'LIB_DIR', str(tmp_path))
    fresh.setenv('CXX', '/bin/false')
    with pytest.warns(UserWarning, match='host path was not built'):
        assert build.build_library() == build.LIB_PATH
