"""csrc/host.cpp against the Python paths it shortens: the same results where it serves a call, None for whatever it does not."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode

import hidet_b200
from hidet_b200 import ffi, native
from hidet_b200.quant import cast_f16_to_u4, w4a16_linear

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def loaded():
    assert native.load() is not None


def _same(x, y):
    if isinstance(x, tuple):
        return len(x) == len(y) and all(_same(p, q) for p, q in zip(x, y))
    return x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and x.device == y.device and torch.equal(x, y)


def _both(monkeypatch, name, native_args, call):
    """The native function serves the operands, and the public call gives the same with it and without it."""
    direct = getattr(native, name)(*native_args)
    assert direct is not None
    public = call()
    with monkeypatch.context() as m:
        m.setattr(native, name, native._unavailable)
        python = call()
    assert _same(direct, python) and _same(public, python)
    return direct


def _weight(k, n, layout='KN', seed=0):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    w = torch.randn((k, n) if layout == 'KN' else (n, k), device='cuda', generator=gen).half() * 0.02
    return hidet_b200.symmetric_quantize(w, 'int8', dims=0 if layout == 'KN' else -1)


def _a(*shape, seed=1):
    return torch.randn(shape, device='cuda', generator=torch.Generator(device='cuda').manual_seed(seed)).half()


@pytest.mark.parametrize('shape,n,layout', [((1, 256), 688, 'KN'), ((2, 3, 512), 256, 'KN'), ((1, 1, 16, 256), 264, 'KN'), ((300, 512), 256, 'KN'), ((7, 256), 258, 'KN'),
                                            ((4, 256), 100, 'NK'), ((64, 512), 512, 'NK'), ((3, 100), 36, 'KN'), ((4, 16384), 256, 'KN')])
@pytest.mark.parametrize('with_out', [False, True])
def test_linear(monkeypatch, shape, n, layout, with_out):
    wq, scale = _weight(shape[-1], n, layout)
    a = _a(*shape)
    hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout=layout)  # makes the stream's scratch
    out = torch.empty(*shape[:-1], n, dtype=torch.float16, device='cuda') if with_out else None
    got = _both(monkeypatch, 'linear', (a, wq, scale, layout, out, None, None, None),
                lambda: hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout=layout, out=out))
    assert not with_out or got is out


@pytest.mark.parametrize('shape,n', [((1, 256), 688), ((2, 3, 512), 256), ((300, 512), 256)])
@pytest.mark.parametrize('bias,residual,activation', [(True, False, None), (False, True, None), (False, False, 'silu_mul'), (True, True, 'silu_mul')])
def test_linear_with_an_epilogue(monkeypatch, shape, n, bias, residual, activation):
    wq, scale = _weight(shape[-1], n)
    a, b = _a(*shape), _a(n, seed=2) if bias else None
    r = _a(*shape[:-1], n // 2 if activation else n, seed=3) if residual else None
    _both(monkeypatch, 'linear', (a, wq, scale, 'KN', None, b, r, activation),
          lambda: hidet_b200.symmetric_quant_matmul(a, wq, scale, bias=b, residual=r, activation=activation))


@pytest.mark.parametrize('rows,cols', [(256, 264), (3, 1001), (1, 1)])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('quant', ['int8', torch.int16])
@pytest.mark.parametrize('dims', [0, 1, -1, -2])
def test_quantize_and_back(monkeypatch, rows, cols, dtype, quant, dims):
    w = _a(rows, cols).to(dtype)
    wq, scale = _both(monkeypatch, 'quantize', (w, quant, dims), lambda: hidet_b200.symmetric_quantize(w, quant, dims=dims))
    _both(monkeypatch, 'dequantize', (wq, scale, dims), lambda: hidet_b200.symmetric_dequantize(wq, scale, dims=dims))


@pytest.mark.parametrize('ids', [torch.tensor([0, 5, -1]), torch.tensor([[3], [2]], dtype=torch.int32), torch.tensor(4)])
def test_embedding_lookup(monkeypatch, ids):
    table, ids = hidet_b200.symmetric_quantize(_a(32, 72), 'int8', dims=-1), ids.cuda()
    _both(monkeypatch, 'take', (*table, ids), lambda: hidet_b200.symmetric_dequantize_take(*table, ids))


@pytest.mark.parametrize('m,k,n,group,with_zp', [(1, 256, 264, 64, True), (40, 512, 128, 128, False), (3, 120, 24, 24, True)])
def test_four_bit_linear(monkeypatch, m, k, n, group, with_zp):
    codes = cast_f16_to_u4(_a(k, n).abs() * 4)
    scale, zeros, a = _a(k // group, n).abs(), _a(k // group, n, seed=2).abs(), _a(m, k, seed=3)
    linear = w4a16_linear('w4', k, n, group, with_zp=with_zp)
    linear(a, codes, scale, zeros)
    _both(monkeypatch, 'w4', (a, codes, scale, zeros if with_zp else None, k, n, group), lambda: linear(a, codes, scale, zeros))


def test_operands_it_leaves_to_the_python_path():
    k, n = 256, 64
    wq, scale = _weight(k, n)
    a = _a(4, k)
    bias, res = _a(n), _a(4, n)
    plain = [a, wq, scale, 'KN', None, None, None, None]
    assert native.linear(*plain) is not None
    double = torch.zeros(8, 2 * k, dtype=torch.float16, device='cuda')
    for at, what in [(0, a.cpu()), (0, double[:4, ::2]), (0, a.float()), (0, a[:, :k - 2].contiguous()), (0, a[0]), (0, a[:0]), (0, 'a'), (1, wq.t()), (1, wq.short()),
                     (1, wq[None]), (1, wq.cpu()), (2, scale[:-2]), (2, scale.float()), (2, scale[None]), (3, 'XY'), (3, 0), (4, res[:2].contiguous()), (4, res.float()),
                     (4, torch.zeros(n, 4, dtype=torch.float16, device='cuda').t()), (5, bias[:-2].contiguous()), (5, bias.float()), (5, bias[None]), (6, res[:, :n // 2].contiguous()),
                     (6, res.float()), (7, 'none'), (7, 'gelu')]:
        args = list(plain)
        args[at] = what
        assert native.linear(*args) is None, (at, what)
    wq_nk, scale_nk = _weight(k, n, 'NK')
    assert native.linear(a, wq_nk, scale_nk, 'NK', None, bias, None, None) is None  # epilogues are for [K, N]
    assert native.linear(a[:, :255].contiguous(), wq[:255].contiguous(), scale, 'KN', None, None, None, None) is None
    w = _a(8, 16)
    assert native.quantize(w, 'int8', 0) is not None
    for args in [(w.cpu(), 'int8', 0), (w.t(), 'int8', 0), (w.double(), 'int8', 0), (w, 'int4', 0), (w, torch.float16, 0), (w, 'int8', [0]), (w, 'int8', 2), (w, 'int8', True),
                 (w[None], 'int8', 0), (w[:0], 'int8', 0)]:
        assert native.quantize(*args) is None, args
    wq2, scale2 = hidet_b200.symmetric_quantize(w, 'int8', dims=0)
    assert native.dequantize(wq2, scale2, 0) is not None
    for args in [(wq2.cpu(), scale2, 0), (wq2, scale2, 1), (wq2, scale2, [0]), (wq2.int(), scale2, 0), (wq2, scale2.double(), 0), (wq2.t(), scale2, 0), (wq2[:0], scale2, 0)]:
        assert native.dequantize(*args) is None, args
    wq2, scale2 = hidet_b200.symmetric_quantize(w, 'int8', dims=-1)
    ids = torch.tensor([1, 2], device='cuda')
    assert native.take(wq2, scale2, ids) is not None
    for args in [(wq2, scale2, ids.cpu()), (wq2, scale2, ids.short()), (wq2, scale2[:-1], ids), (wq2.float(), scale2, ids), (wq2, scale2, ids[:0])]:
        assert native.take(*args) is None, args
    codes, s4, a4 = torch.zeros(128, 8, dtype=torch.int32, device='cuda'), _a(2, 64), _a(3, 128)
    w4a16_linear('w4', 128, 64, 64, with_zp=False)(a4, codes, s4)
    good = [a4, codes, s4, None, 128, 64, 64]
    assert native.w4(*good) is not None
    for at, what in [(0, a4.float()), (0, a4[:, :64].contiguous()), (0, _a(3 * 128 + 1)[1:].view(3, 128)), (0, a4.cpu()), (1, codes[:64]), (1, codes.t()), (2, s4[:1]), (2, s4.float()),
                     (3, s4[:1]), (3, s4.t()), (4, 64), (6, 0), (6, 100)]:
        args = list(good)
        args[at] = what
        assert native.w4(*args) is None, (at, what)


def test_scratch_that_does_not_exist_yet_is_left_to_the_python_path():
    wq, scale = _weight(16384, 256)
    a = _a(4, 16384)
    assert ffi.func('b200q_qlinear_workspace_bytes')(4, 256, 16384, ffi.LAYOUT_KN) > 0
    want = hidet_b200.symmetric_quant_matmul(a, wq, scale)
    stream = torch.cuda.ExternalStream(torch.cuda.Stream(priority=-1).cuda_stream)
    hidet_b200.runtime.workspaces.clear()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        plain = (a, wq, scale, 'KN', None, None, None, None)
        assert native.linear(*plain) is None
        assert torch.equal(hidet_b200.symmetric_quant_matmul(a, wq, scale), want)
        assert torch.equal(native.linear(*plain), want)
        stream.synchronize()
    assert native.linear(*plain) is None  # the scratch is that stream's
    assert torch.equal(hidet_b200.symmetric_quant_matmul(a, wq, scale), want)


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


def test_fake_results_and_wrapped_tensors_are_refused_as_before():
    a, (wq, scale) = _a(4, 256), _weight(256, 64)
    with FakeTensorMode(), pytest.raises(ffi.BackendException, match='null output'):
        hidet_b200.symmetric_quant_matmul(a, wq, scale)
    with pytest.raises(RuntimeError, match='storage'):
        torch.vmap(lambda w: hidet_b200.symmetric_quantize(w, 'int8', dims=0)[0])(_a(2, 8, 16))
