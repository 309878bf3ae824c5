"""Operands that the kernel in front writes, where the kernels launched as programmatic dependents promise to wait for its end: 4-bit weights,
int8 weights whose rows are not multiples of 16 bytes, int8 weights of the kernels for more than a few rows and of 17 to 24 rows on 6 MB and more, the
scales of every weight, and all operands of the quantize, dequantize and lookup kernels.  (Otherwise the small-M int8 kernel asks for the codes of its
weight earlier by contract, and is tested behind this library's own producers only.)"""
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


@pytest.fixture(scope='module')
def late_copy_everywhere(nvcc_library):
    """late_copy by a kernel that fills every SM's first-level cache with the old values before it lets its dependents start."""
    f = nvcc_library('late_copy.cu').late_copy_everywhere
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def copy(dst, src):
        assert dst.shape == src.shape and dst.dtype == src.dtype and dst.numel() * dst.element_size() % 4 == 0
        assert f(dst.data_ptr(), src.data_ptr(), dst.numel() * dst.element_size() // 4, 40000, sms, torch.cuda.current_stream().cuda_stream) == 0

    return copy


def _bytes(*tensors):
    return torch.cat([t.contiguous().view(torch.uint8).reshape(-1) for t in tensors])


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
    """The packing and quantizing kernels let nothing start before their end: the next call may read what they write into the same buffers."""
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


# whole vectors and other widths; rows for a warp, for a CTA (24 to 96 KB), and longer; bases off a vector's boundary
SHAPES = [(300, 64), (300, 61), (64, 13000), (64, 13001), (6, 50000), (12, 50001), (4000, 8), (7, 12)]


@pytest.mark.parametrize('rows,cols', SHAPES)
@pytest.mark.parametrize('dims', [0, -1])
@pytest.mark.parametrize('dtype', [torch.float16, torch.float32])
@pytest.mark.parametrize('everywhere', [False, True])
def test_quantized_values_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, late_copy_everywhere, rows, cols, dims, dtype, everywhere):
    gen = torch.Generator(device='cuda').manual_seed(rows + cols)
    weights = [(torch.randn(rows, cols, device='cuda', generator=gen).to(dtype),) for _ in range(2)]
    _check(late_copy_everywhere if everywhere else late_copy, weights, lambda w: _bytes(*hidet_b200.symmetric_quantize(w, 'int8', dims=dims)))


@pytest.mark.parametrize('rows,cols', SHAPES)
@pytest.mark.parametrize('dims', [0, -1])
@pytest.mark.parametrize('dtype,quant', [(torch.float16, torch.int8), (torch.float32, torch.int16)])
@pytest.mark.parametrize('everywhere', [False, True])
def test_restored_values_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, late_copy_everywhere, rows, cols, dims, dtype, quant, everywhere):
    gen = torch.Generator(device='cuda').manual_seed(rows + cols)
    padded = (cols if dims == 0 else rows) // 4 * 4 + 4   # whole words to copy
    weights = [(torch.randint(-127, 128, (rows, (cols + 3) // 4 * 4), device='cuda', generator=gen).to(quant),
                torch.rand(padded, device='cuda', generator=gen).to(dtype)) for _ in range(2)]

    def call(codes, scale):
        # the first rows * cols codes of the buffer
        return _bytes(hidet_b200.symmetric_dequantize(codes.view(-1)[:rows * cols].view(rows, cols), scale[:cols if dims == 0 else rows], dims=dims))

    _check(late_copy_everywhere if everywhere else late_copy, weights, call)


@pytest.mark.parametrize('dim', [64, 61])
@pytest.mark.parametrize('index', [torch.int32, torch.int64])
@pytest.mark.parametrize('everywhere', [False, True])
def test_lookups_may_read_the_result_of_a_kernel_that_triggers_early(late_copy, late_copy_everywhere, dim, index, everywhere):
    gen = torch.Generator(device='cuda').manual_seed(dim)
    vocab = 400
    weights = [(torch.randint(0, vocab, (70,), device='cuda', generator=gen).to(index), torch.randint(-127, 128, (vocab, dim), device='cuda', generator=gen).to(torch.int8),
                torch.rand(vocab, device='cuda', generator=gen).half()) for _ in range(2)]
    _check(late_copy_everywhere if everywhere else late_copy, weights, lambda ids, table, scale: _bytes(hidet_b200.symmetric_dequantize_take(table, scale, ids)))


@pytest.mark.parametrize('m,k,n,kind', [(17, 2048, 3072, 0), (24, 2048, 3072, 0), (100, 1024, 1024, 1), (1100, 1024, 4096, 2)])
@pytest.mark.parametrize('layout', ['KN', 'NK'])
def test_weights_of_more_than_16_rows_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, large_kernels, m, k, n, kind, layout):
    out = (ctypes.c_int * 3)()
    large_kernels.plan(m, n, k, 0, out)
    assert out[0] == kind
    gen = torch.Generator(device='cuda').manual_seed(m)
    a = torch.randn(m, k, device='cuda', generator=gen).half()
    weights = [(torch.randint(-127, 128, (k, n) if layout == 'KN' else (n, k), device='cuda', generator=gen, dtype=torch.int8),
                torch.rand(n, device='cuda', generator=gen).mul_(1e-2).half()) for _ in range(2)]
    _check(late_copy, weights, lambda wq, scale: hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout=layout))


# in front: the three kernels of the linears, each with SMs to spare
@pytest.mark.parametrize('rows,k,n', [(8, 4096, 1024), (100, 4096, 1024), (520, 4096, 3072)])
@pytest.mark.parametrize('dims', [0, -1])
def test_quantize_and_dequantize_may_read_the_result_of_the_linear_in_front(rows, k, n, dims):
    gen = torch.Generator(device='cuda').manual_seed(rows)
    wq = torch.randint(-127, 128, (k, n), device='cuda', generator=gen, dtype=torch.int8)
    ones = torch.full((n,), 1e-4, device='cuda').half()
    fronts = [torch.randn(rows, k, device='cuda', generator=gen).half() for _ in range(2)]
    codes = torch.randint(-127, 128, (rows, n) if dims == 0 else (n, rows), device='cuda', generator=gen, dtype=torch.int8)
    buffer = torch.zeros(rows, n, dtype=torch.float16, device='cuda')

    def all_three(x, between):
        hidet_b200.symmetric_quant_matmul(x, wq, ones, out=buffer)
        between()
        first = hidet_b200.symmetric_quantize(buffer, 'int8', dims=dims)
        hidet_b200.symmetric_quant_matmul(x, wq, ones, out=buffer)
        between()
        return _bytes(*first, hidet_b200.symmetric_dequantize(codes, buffer[rows - 1], dims=dims))   # a row of the result as scales

    want = [all_three(x, torch.cuda.synchronize) for x in fronts]
    torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    for i in range(12):
        assert torch.equal(all_three(fronts[i % 2], lambda: None), want[i % 2])
    assert ffi.func('b200q_check_status')() == ffi.OK


# calls beyond 24 rows that the small-M kernel would serve as fast
@pytest.mark.parametrize('m,k,n', [(56, 1536, 6144), (64, 1536, 6144), (51, 1680, 5776), (49, 1536, 6144)])
@pytest.mark.parametrize('layout', ['KN', 'NK'])
def test_weights_beyond_24_rows_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, m, k, n, layout):
    gen = torch.Generator(device='cuda').manual_seed(m)
    a = torch.randn(m, k, device='cuda', generator=gen).half()
    weights = [(torch.randint(-127, 128, (k, n) if layout == 'KN' else (n, k), device='cuda', generator=gen, dtype=torch.int8),
                torch.rand(n, device='cuda', generator=gen).mul_(1e-2).half()) for _ in range(2)]
    _check(late_copy, weights, lambda wq, scale: hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout=layout))


# the kernels that take odd widths in aligned vectors, which they do from more elements on than the shapes above have
@pytest.mark.parametrize('dims', [0, -1])
@pytest.mark.parametrize('dtype,quant', [(torch.float16, torch.int8), (torch.float32, torch.int16)])
def test_odd_widths_in_vectors_may_be_the_result_of_a_kernel_that_triggers_early(late_copy, dims, dtype, quant):
    rows, cols = 3072, 1026 + (dtype == torch.float16)   # 1026 is not a multiple of four
    gen = torch.Generator(device='cuda').manual_seed(cols)
    weights = [(torch.randn(rows, cols, device='cuda', generator=gen).to(dtype),) for _ in range(2)]
    _check(late_copy, weights, lambda w: _bytes(*hidet_b200.symmetric_quantize(w, 'int8', dims=dims)))
    codes = [(torch.randint(-127, 128, (rows, cols), device='cuda', generator=gen).to(quant), torch.rand(cols // 4 * 4 + 4 if dims == 0 else rows, device='cuda', generator=gen).to(dtype))
             for _ in range(2)]
    _check(late_copy, codes, lambda q, s: _bytes(hidet_b200.symmetric_dequantize(q, s[:cols if dims == 0 else rows], dims=dims)))
