"""Operands that the kernel in front writes, where the quantized linears promise to wait for its end: 4-bit weights, int8
weights whose rows are not multiples of 16 bytes, and the scales of every weight.  (The small-M int8 kernel asks for the codes
of its weight earlier by contract, and is tested behind this library's own producers only.)"""
import ctypes

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi
from hidet_b200.quant import cast_f16_to_u4, w4a16_linear

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def late_copy(nvcc_library):
    f = nvcc_library('late_copy.cu').late_copy
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]

    def copy(dst, src):
        assert dst.shape == src.shape and dst.dtype == src.dtype and dst.numel() * dst.element_size() % 4 == 0
        assert f(dst.data_ptr(), src.data_ptr(), dst.numel() * dst.element_size() // 4, 40000, torch.cuda.current_stream().cuda_stream) == 0

    return copy


def _check(late_copy, weights, call):
    """Each of `weights` is copied late into the same buffers, tensor by tensor, right in front of the call that reads them."""
    want = [call(*w) for w in weights]
    torch.cuda.synchronize()
    for which in range(len(weights[0])):
        mine = [t.clone() for t in weights[0]]
        expect = [call(*(w[j] if j == which else weights[0][j] for j in range(len(mine)))) for w in weights]
        torch.cuda.synchronize()
        got = []
        for w in weights * 3:
            late_copy(mine[which], w[which])
            got.append(call(*mine))
        assert not torch.equal(want[0], want[1])
        for i, g in enumerate(got):
            assert torch.equal(g, expect[i % len(weights)])
    assert ffi.func('b200q_check_status')() == ffi.OK


@pytest.mark.parametrize('m,k,n', [(1, 512, 1536), (8, 256, 1000), (16, 512, 264), (33, 256, 512)])
def test_four_bit_weights_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, m, k, n):
    gen = torch.Generator(device='cuda').manual_seed(k + n)
    a = torch.randn(m, k, device='cuda', generator=gen).half()
    weights = [(cast_f16_to_u4(torch.randint(0, 16, (k, n), device='cuda', generator=gen).half()),
                torch.rand(k // 128, n, device='cuda', generator=gen).half(), torch.rand(k // 128, n, device='cuda', generator=gen).mul_(15).half()) for _ in range(2)]
    linear = w4a16_linear('w4a16', k, n, 128)
    _check(late_copy, weights, lambda codes, scale, zeros: linear(a, codes, scale, zeros))


@pytest.mark.parametrize('m,k,n', [(1, 512, 514), (8, 256, 1004), (16, 512, 222)])
def test_weights_of_odd_rows_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, m, k, n):
    gen = torch.Generator(device='cuda').manual_seed(k + n)
    a = torch.randn(m, k, device='cuda', generator=gen).half()
    weights = [hidet_b200.symmetric_quantize(torch.randn(k, n, device='cuda', generator=gen).half() * 0.02, 'int8', dims=0) for _ in range(2)]
    _check(late_copy, weights, lambda wq, scale: hidet_b200.symmetric_quant_matmul(a, wq, scale))


@pytest.mark.parametrize('m', [1, 16, 48])
def test_weights_rewritten_by_this_library_between_calls(m):
    """The packing and quantizing kernels are ordinary: the next call may read what they write into the same buffers."""
    k, n = 512, 1024
    gen = torch.Generator(device='cuda').manual_seed(m)
    a = torch.randn(m, k, device='cuda', generator=gen).half()
    linear = w4a16_linear('w4a16', k, n, 128, with_zp=False)
    scale4 = torch.rand(k // 128, n, device='cuda', generator=gen).half()
    codes = [torch.randint(0, 16, (k, n), device='cuda', generator=gen).half() for _ in range(2)]
    floats = [torch.randn(k, n, device='cuda', generator=gen).half() * 0.02 for _ in range(2)]
    want4 = [linear(a, cast_f16_to_u4(c), scale4) for c in codes]
    want8 = [hidet_b200.symmetric_quant_matmul(a, *hidet_b200.symmetric_quantize(w, 'int8', dims=0)) for w in floats]
    packed = torch.empty(k, n // 8, dtype=torch.int32, device='cuda')
    wq, scale8 = torch.empty(k, n, dtype=torch.int8, device='cuda'), torch.empty(n, dtype=torch.float16, device='cuda')
    stream = torch.cuda.current_stream().cuda_stream
    got4, got8 = [], []
    for i in range(6):
        ffi.func('b200q_u4_pack')(codes[i % 2].data_ptr(), packed.data_ptr(), k, n, stream)
        got4.append(linear(a, packed, scale4))
        ffi.func('b200q_symmetric_quantize')(floats[i % 2].data_ptr(), wq.data_ptr(), scale8.data_ptr(), k, n, ffi.F16, ffi.I8, 0, stream)
        got8.append(hidet_b200.symmetric_quant_matmul(a, wq, scale8))
    for i in range(6):
        assert torch.equal(got4[i], want4[i % 2]) and torch.equal(got8[i], want8[i % 2])


# in front: the small-M kernel, the mid-M one and the one on SM pairs, each with SMs to spare, so that the launch behind them starts early
@pytest.mark.parametrize('rows,k,n', [(8, 4096, 1024), (100, 4096, 1024), (520, 4096, 3072)])
@pytest.mark.parametrize('m', [1, 6, 16])
@pytest.mark.parametrize('layout', ['KN', 'NK'])
def test_scales_may_be_the_result_of_the_linear_in_front(rows, k, n, m, layout):
    gen = torch.Generator(device='cuda').manual_seed(rows + m)
    codes = torch.randint(-127, 128, (k, n), device='cuda', generator=gen, dtype=torch.int8)
    ones = torch.full((n,), 1e-4, device='cuda').half()
    fronts = [torch.randn(rows, k, device='cuda', generator=gen).half() for _ in range(2)]
    a = torch.randn(m, 4096, device='cuda', generator=gen).half()
    wq = torch.randint(-127, 128, (4096, n) if layout == 'KN' else (n, 4096), device='cuda', generator=gen, dtype=torch.int8)
    buffer = torch.zeros(rows, n, dtype=torch.float16, device='cuda')

    def both(x, between):
        hidet_b200.symmetric_quant_matmul(x, codes, ones, out=buffer)
        between()
        return hidet_b200.symmetric_quant_matmul(a, wq, buffer[rows - 1], weight_layout=layout)

    want = [both(x, torch.cuda.synchronize) for x in fronts]
    torch.cuda.synchronize()
    got = [both(fronts[i % 2], lambda: None) for i in range(12)]
    assert not torch.equal(want[0], want[1])
    for i, g in enumerate(got):
        assert torch.equal(g, want[i % 2])
    assert ffi.func('b200q_check_status')() == ffi.OK
