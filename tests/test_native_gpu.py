"""csrc/host.cpp against the Python paths it shortens."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import hidet_b200
from hidet_b200 import native

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def loaded():
    assert native.load() is not None


def _weight(k, n, layout='KN', seed=0):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    w = torch.randn((k, n) if layout == 'KN' else (n, k), device='cuda', generator=gen).half() * 0.02
    return hidet_b200.symmetric_quantize(w, 'int8', dims=0 if layout == 'KN' else -1)


def _a(*shape, seed=1):
    return torch.randn(shape, device='cuda', generator=torch.Generator(device='cuda').manual_seed(seed)).half()


def test_dispatch_modes_see_what_they_saw():
    class Names(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(func.name())
            return func(*args, **(kwargs or {}))

    wq, scale = _weight(256, 64)
    a = _a(4, 256)
    want = hidet_b200.symmetric_quant_matmul(a, wq, scale)
    with Names() as names:
        assert native.linear(a, wq, scale, 'KN', None, None, None, None) is None
        assert native.quantize(a, 'int8', 0) is None and native.dequantize(wq, scale, 0) is None
        got = hidet_b200.symmetric_quant_matmul(a, wq, scale)
    assert torch.equal(got, want) and any('empty' in name for name in names.seen)


def test_wrapped_tensors_are_refused_as_before():
    with pytest.raises(RuntimeError, match='storage'):
        torch.vmap(lambda w: hidet_b200.symmetric_quantize(w, 'int8', dims=0)[0])(_a(2, 8, 16))
