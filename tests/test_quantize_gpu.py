"""symmetric_quantize / symmetric_dequantize on the GPU against the CPU oracle: bit-exact."""
import numpy as np
import pytest
import torch

from conftest import seeded_weight

import hidet_b200
import oracle

pytestmark = pytest.mark.gpu


def _gpu_quantize(w_np, quant_type, dims):
    w = torch.from_numpy(w_np).cuda()
    wq, scale = hidet_b200.symmetric_quantize(w, quant_type, dims=dims)
    torch.cuda.synchronize()
    return wq.cpu().numpy(), scale.cpu().numpy()


def _assert_same(w_np, quant_type, dims, what):
    wq, scale = _gpu_quantize(w_np, quant_type, dims)
    wq_o, scale_o = oracle.symmetric_quantize(w_np, quant_type, dims)
    assert wq.dtype == wq_o.dtype and wq.shape == wq_o.shape and scale.shape == scale_o.shape, what
    bits = np.uint16 if w_np.dtype == np.float16 else np.uint32
    assert np.array_equal(scale.view(bits), scale_o.view(bits)), '{}: {} scale words differ'.format(
        what, int((scale.view(bits) != scale_o.view(bits)).sum()))
    assert np.array_equal(wq, wq_o), '{}: {} of {} codes differ'.format(what, int((wq != wq_o).sum()), wq.size)
    return wq, scale


# shapes and dims of the reference's tests (tests/operators_core/test_quantization.py:21-36,
# tests/operators_core/test_symmetric_quant.py:19-26) plus ragged and projection-like ones
@pytest.mark.parametrize('shape', [(32, 32), (64, 64), (256, 192), (67, 45), (1, 8), (8, 1), (3, 1000), (1000, 24), (513, 136)])
@pytest.mark.parametrize('dims', [0, -1])
@pytest.mark.parametrize('quant_type', ['int8', 'int16'])
def test_quantize_f16_bit_exact(shape, dims, quant_type):
    rng = np.random.default_rng(hash((shape, dims)) % 2**31)
    w = rng.standard_normal(shape).astype(np.float16)
    _assert_same(w, quant_type, dims, 'randn {} dims={} {}'.format(shape, dims, quant_type))


@pytest.mark.parametrize('k,n', [(4096, 4096), (4096, 11008), (11008, 4096)])
def test_quantize_projection_shapes_bit_exact(k, n):
    w = seeded_weight(k, n, seed=k + n)
    wq, scale = _assert_same(w, 'int8', 0, 'weight [{}, {}]'.format(k, n))
    assert int(np.abs(wq.astype(np.int32)).max()) == 127


def test_quantize_row_wise_long_rows():
    w = seeded_weight(300, 11008, seed=9)
    _assert_same(w, 'int8', -1, 'row-wise [300, 11008]')


def test_quantize_edge_values():
    rng = np.random.default_rng(11)
    w = (rng.standard_normal((128, 64)) * 0.02).astype(np.float16)
    w[:, 0] = 0.0                       # scale 0 -> 0/0
    w[:, 1] = np.float16(-0.0)          # all negative zero
    w[:, 2] = np.abs(w[:, 2])           # one sign only
    w[:, 3] = np.float16(6e-8)          # smallest subnormal: the scale underflows to zero, w/0 = inf
    w[:, 4] = np.float16(65504.0)       # largest finite value
    w[5, 5] = np.float16(30000.0)       # an outlier that owns the scale
    w[:, 6] = np.float16(1e-3)          # a scale in the range where the division takes its correction step
    w[:, 7] = (np.arange(128) % 7 - 3).astype(np.float16)   # many exact ties
    for dims in (0, -1):
        _assert_same(w, 'int8', dims, 'edge values dims={}'.format(dims))
        _assert_same(w, 'int16', dims, 'edge values dims={} int16'.format(dims))


def special_value_weight(rows):
    """[rows, 64] f16 whose first columns hold NaN, infinities and signed zeros in the mixes that decide the
    absmax: abs is `(0 <= w) ? w : -w` and max is __hmax, so a NaN is skipped, -0 stays -0 and loses to +0."""
    rng = np.random.default_rng(14)
    w = (rng.standard_normal((rows, 64)) * 0.02).astype(np.float16)
    nan, inf = np.float16(np.nan), np.float16(np.inf)
    w[:, 0] = nan                                   # nothing but NaN: the absmax stays at the lowest finite value
    w[:, 1] = np.float16(-0.0); w[7, 1] = nan       # -0 and a NaN: absmax -0
    w[:, 2] = np.float16(-0.0); w[rows - 1, 2] = np.float16(0.0)   # one +0 among -0: absmax +0
    w[5, 3] = nan; w[rows // 2, 3] = -nan           # NaN of both signs inside ordinary values
    w[3, 4] = inf                                   # +inf owns the scale
    w[rows - 2, 5] = -inf                           # -inf does
    w[:, 6] = -np.abs(w[:, 6]) - np.float16(1e-3)   # negative values only
    w[:, 7] = np.float16(-65504.0)                  # the lowest finite value itself
    w[:, 8] = np.float16(-0.0)                      # -0 only
    w[:, 9] = np.float16(-0.0); w[1, 9] = np.float16(-6e-8)   # -0 and the negative subnormal next to it
    return w


@pytest.mark.parametrize('rows', [128, 1100])
def test_quantize_nan_inf_and_signed_zero_columns(rows):
    w = special_value_weight(rows)
    # an odd column count takes the element-wise kernels, a multiple of eight the packed ones: the same columns
    # must come out the same
    wq_v, scale_v = _gpu_quantize(w, 'int8', 0)
    wq_e, scale_e = _gpu_quantize(np.ascontiguousarray(w[:, :63]), 'int8', 0)
    assert np.array_equal(scale_v[:63].view(np.uint16), scale_e.view(np.uint16)) and np.array_equal(wq_v[:, :63], wq_e)
    for dims in (0, -1):
        _assert_same(w, 'int8', dims, 'special values rows={} dims={}'.format(rows, dims))
        _assert_same(w, 'int16', dims, 'special values rows={} dims={} int16'.format(rows, dims))
    wt = np.ascontiguousarray(w.T)          # the same columns as rows of the row-wise form
    _assert_same(wt, 'int8', -1, 'special values transposed rows={}'.format(rows))


def test_quantize_tie_heavy_grid():
    # values on a coarse grid make w / scale land exactly on .5 in many places
    rng = np.random.default_rng(12)
    w = (rng.integers(-254, 255, size=(512, 256)) / 2.0).astype(np.float16)
    w[0, :] = 127.0
    wq, _ = _assert_same(w, 'int8', 0, 'tie grid')
    # ties to even: 0.5 -> 0, 1.5 -> 2, 2.5 -> 2
    assert np.array_equal(wq[w == 0.5], np.zeros((w == 0.5).sum(), dtype=np.int8))
    assert np.array_equal(wq[w == 2.5], np.full((w == 2.5).sum(), 2, dtype=np.int8))


def test_quantize_unaligned_and_batched_views():
    rng = np.random.default_rng(13)
    base = rng.standard_normal((65, 70)).astype(np.float16)
    w = torch.from_numpy(base).cuda()[1:, 3:67]  # non-contiguous view, odd offsets
    wq, scale = hidet_b200.symmetric_quantize(w, 'int8', dims=0)
    wq_o, scale_o = oracle.symmetric_quantize(np.ascontiguousarray(base[1:, 3:67]), 'int8', 0)
    assert np.array_equal(wq.cpu().numpy(), wq_o) and np.array_equal(scale.cpu().numpy().view(np.uint16), scale_o.view(np.uint16))
    w3 = rng.standard_normal((4, 6, 40)).astype(np.float16)
    _assert_same(w3, 'int8', -1, '3-D last dim')
    _assert_same(w3, 'int8', 0, '3-D first dim')


@pytest.mark.parametrize('dims', [0, -1])
def test_quantize_f32_against_ieee_oracle(dims):
    # f32 on the GPU divides with the approximate division the reference's build flags select
    # (-prec-div=false), which is within 2 ulp of the IEEE quotient: scales agree to 2 ulp, codes differ
    # by at most one step where a quotient sits on a rounding boundary.
    rng = np.random.default_rng(14)
    w = (rng.standard_normal((300, 200)) * 0.02).astype(np.float32)
    wq, scale = _gpu_quantize(w, 'int8', dims)
    wq_o, scale_o = oracle.symmetric_quantize(w, 'int8', dims)
    d = scale.view(np.uint32).astype(np.int64) - scale_o.view(np.uint32).astype(np.int64)
    assert np.abs(d).max() <= 2
    diff = wq.astype(np.int32) - wq_o.astype(np.int32)
    assert np.abs(diff).max() <= 1 and (diff != 0).mean() < 1e-3


@pytest.mark.parametrize('dims', [0, -1])
def test_quantize_bf16_round_trip(dims):
    # tests/operators_core/test_quantization.py:21-36 runs bfloat16 too, with atol = rtol = 1e-1
    g = torch.Generator().manual_seed(15)
    w = torch.randn(64, 64, generator=g).to(torch.bfloat16).cuda()
    for qt in ('int8', 'int16'):
        wq, scale = hidet_b200.symmetric_quantize(w, qt, dims=dims)
        wd = hidet_b200.symmetric_dequantize(wq, scale, dims=dims)
        assert wd.dtype == torch.bfloat16
        assert torch.allclose(wd.float(), w.float(), atol=1e-1, rtol=1e-1)


@pytest.mark.parametrize('shape', [(32, 32), (64, 64), (67, 45), (4096, 4096), (513, 136)])
@pytest.mark.parametrize('dims', [0, -1])
def test_dequantize_bit_exact_and_round_trip(shape, dims):
    w = seeded_weight(shape[0], shape[1], seed=21, std=1.0)
    wq_o, scale_o = oracle.symmetric_quantize(w, 'int8', dims)
    wd = hidet_b200.symmetric_dequantize(torch.from_numpy(wq_o).cuda(), torch.from_numpy(scale_o).cuda(), dims=dims)
    wd_o = oracle.symmetric_dequantize(wq_o, scale_o, dims)
    assert np.array_equal(wd.cpu().numpy().view(np.uint16), wd_o.view(np.uint16))
    # the reference's own acceptance test: quantize -> dequantize within atol = rtol = 1e-1
    assert np.allclose(wd_o.astype(np.float32), w.astype(np.float32), atol=1e-1, rtol=1e-1)


def test_quantize_commutes_with_column_sharding():
    w = seeded_weight(1024, 512, seed=22)
    wq, scale = _gpu_quantize(w, 'int8', 0)
    for g in (2, 4, 8):
        step = 512 // g
        for r in range(g):
            wq_r, scale_r = _gpu_quantize(np.ascontiguousarray(w[:, r * step:(r + 1) * step]), 'int8', 0)
            assert np.array_equal(wq_r, wq[:, r * step:(r + 1) * step])
            assert np.array_equal(scale_r.view(np.uint16), scale[r * step:(r + 1) * step].view(np.uint16))


def test_quantize_rejects_bad_arguments():
    w = torch.zeros(8, 8, dtype=torch.float16, device='cuda')
    with pytest.raises(ValueError):
        hidet_b200.symmetric_quantize(w, 'int4', dims=0)
    with pytest.raises(ValueError):
        hidet_b200.symmetric_quantize(w.to(torch.int32), 'int8', dims=0)
    with pytest.raises(ValueError):
        hidet_b200.symmetric_quantize(w, 'int8', dims=2)
    wq, scale = hidet_b200.symmetric_quantize(w, 'int8', dims=0)
    with pytest.raises(ValueError):
        hidet_b200.symmetric_dequantize(wq, scale[:4], dims=0)


def test_quotient_of_halves_is_cuda_s_for_every_pair(nvcc_library):
    """The quantize kernels take w / scale as the rounded reciprocal times w; all 2^32 pairs, with the flags they are compiled with."""
    import ctypes

    from hidet_b200.build import PER_SOURCE_FLAGS

    f = nvcc_library('half_quotient.cu', *PER_SOURCE_FLAGS['quantize.cu']).half_quotient_mismatches
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    mismatches = torch.zeros(1, dtype=torch.int64, device='cuda')
    assert f(mismatches.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert mismatches.item() == 0


def test_quotient_of_bfloat16_is_cuda_s(nvcc_library):
    """As above for bfloat16, over every divisor that is taken as its reciprocal."""
    import ctypes

    from hidet_b200.build import PER_SOURCE_FLAGS

    f = nvcc_library('bf16_quotient.cu', *PER_SOURCE_FLAGS['quantize.cu']).bf16_quotient_mismatches
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    mismatches = torch.zeros(1, dtype=torch.int64, device='cuda')
    assert f(mismatches.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert mismatches.item() == 0


@pytest.mark.parametrize('rows,cols', [(128, 64), (1100, 72), (37, 4104)])
def test_quantize_bf16_bits(rows, cols):
    """bfloat16 with special values: the packed kernels (columns a multiple of eight) give what the element-wise ones (an odd
    count) do, and the definition in f32 steps where all is finite."""
    g = torch.Generator().manual_seed(rows)
    w = torch.randn(rows, cols, generator=g).mul_(0.02).to(torch.bfloat16)
    finite = w.clone()
    nan, inf = float('nan'), float('inf')
    w[:, 0] = nan
    w[:, 1] = -0.0; w[7, 1] = nan
    w[:, 2] = -0.0; w[rows - 1, 2] = 0.0
    w[5, 3] = nan
    w[3, 4] = inf
    w[rows - 2, 5] = -inf
    w[:, 6] = -w[:, 6].abs() - 1e-3
    w[:, 7] = 3.3895313892515355e38
    w[:, 8] = 1e-40                     # below the normal numbers
    w[:, 9] = 1.1754943508222875e-38; w[0, 9] = 5e-39   # the smallest normal number: the scale is below
    w[:, 10] = 1.5e-36; w[0, 10] = 1e-39  # a scale next to the smallest normal number
    w[:, 11] = torch.arange(rows) % 255 - 127.0   # exact ties
    for dims in (0, -1):
        both = w if dims == 0 else w.t().contiguous()
        odd = both[:, :-1].contiguous() if dims == 0 else torch.cat([both, both[:, :1]], 1)
        q, s = hidet_b200.symmetric_quantize(both.cuda(), 'int8', dims=dims)
        qo, so = hidet_b200.symmetric_quantize(odd.cuda(), 'int8', dims=dims)
        n = qo.shape[1] if dims == 0 else q.shape[1]
        assert torch.equal(s[:len(so)].view(torch.int16).cpu(), so.view(torch.int16).cpu())
        assert torch.equal(q[:, :n].cpu(), qo[:, :n].cpu())
        q, s = hidet_b200.symmetric_quantize(finite.cuda(), 'int8', dims=dims)
        want_s = (finite.abs().amax(dim=dims).float() / 127).to(torch.bfloat16)
        assert torch.equal(s.cpu(), want_s)
        quotient = (finite.float() / want_s.float().unsqueeze(dims)).to(torch.bfloat16)
        inside = quotient.float().abs() <= 127   # (a scale rounded down leaves quotients of 127.5: what the conversion makes of 128 is compared above)
        assert torch.equal(q.cpu()[inside], quotient.float().round().to(torch.int8)[inside])


def _bits(t):
    return t if t.dtype in (torch.int8, torch.int16) else t.view(torch.int16 if t.element_size() == 2 else torch.int32)


# Widths that are not whole vectors against the same matrix with its rows filled up, which the kernels for whole vectors take (and the oracle
# pins): with NaN, which the maximum skips.  Rows that begin everywhere inside a vector, rows shorter than a panel and longer than what a warp
# keeps, fewer rows than a group, a last vector that would reach past the matrix, slices that do not fit shared memory.
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('quant_type', ['int8', 'int16'])
@pytest.mark.parametrize('rows,cols', [(1, 9), (7, 9), (3, 57), (64, 63), (513, 113), (2001, 1027), (4099, 62), (260, 517), (19, 24581), (26111, 58)])
def test_widths_that_are_not_whole_vectors(rows, cols, quant_type, dtype):
    g = torch.Generator(device='cuda').manual_seed(rows + cols)
    wide = torch.full((rows, (cols + 15) // 8 * 8), float('nan'), device='cuda', dtype=dtype)
    wide[:, :cols] = torch.randn(rows, cols, device='cuda', generator=g).mul_(0.02).to(dtype)
    wide[0, 0], wide[rows - 1, cols - 1], wide[rows // 2, cols // 2] = float('nan'), float('inf'), -0.0
    wide[rows // 3, :cols] = -0.0
    wide[:, 4] = -wide[:, 4].abs()
    w = wide[:, :cols].contiguous()
    for dims in (0, -1):
        wq, scale = hidet_b200.symmetric_quantize(w, quant_type, dims=dims)
        wq_w, scale_w = hidet_b200.symmetric_quantize(wide, quant_type, dims=dims)
        assert torch.equal(_bits(scale), _bits(scale_w)[:cols] if dims == 0 else _bits(scale_w))
        assert torch.equal(wq, wq_w[:, :cols])
        scale = torch.rand(scale.shape, device='cuda', generator=g).to(dtype)
        scale_w = scale if dims == -1 else torch.cat([scale, scale.new_ones(wide.shape[1] - cols)])
        back = hidet_b200.symmetric_dequantize(wq, scale, dims=dims)
        assert torch.equal(_bits(back), _bits(hidet_b200.symmetric_dequantize(wq_w, scale_w, dims=dims)[:, :cols].contiguous()))


def test_slices_that_fill_the_default_shared_memory():
    """Slices of a panel between 47 and 48 KB, with the static arrays above what a launch gets unasked: in a process of its own, where no
    larger slice has asked for more."""
    import os
    import subprocess
    import sys

    code = ("import torch, hidet_b200\n"
            "w = torch.randn(6144, 64, device='cuda').half()\n"
            "wq, scale = hidet_b200.symmetric_quantize(w, 'int8', dims=0)\n"
            "rows = [hidet_b200.symmetric_quantize(w.t().contiguous(), 'int8', dims=-1)]\n"
            "assert torch.equal(wq, rows[0][0].t()) and torch.equal(scale, rows[0][1])\n")
    subprocess.run([sys.executable, '-c', code], check=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


# sizes beyond the lines from which on odd widths go in aligned vectors: restored from 3 Mi elements (96 columns) and 16 Mi (48), quantized per row
# from four rows an SM (512 bytes) and eight; below and above each
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('quant_type', ['int8', 'int16'])
@pytest.mark.parametrize('rows,cols', [(3063, 1027), (3062, 1027), (32769, 97), (33150, 95), (6, 600001), (350003, 49), (342393, 49), (593, 301), (591, 301), (1185, 9), (1183, 9), (2003, 12001)])
def test_widths_in_vectors_and_element_by_element(rows, cols, quant_type, dtype):
    g = torch.Generator(device='cuda').manual_seed(rows + cols)
    wide = torch.full((rows, (cols + 15) // 8 * 8), float('nan'), device='cuda', dtype=dtype)
    wide[:, :cols] = torch.randn(rows, cols, device='cuda', generator=g).mul_(0.02).to(dtype)
    wide[0, 0], wide[rows - 1, cols - 1], wide[rows // 2, cols // 2] = float('nan'), float('inf'), -0.0
    w = wide[:, :cols].contiguous()
    for dims in (0, -1):
        wq, scale = hidet_b200.symmetric_quantize(w, quant_type, dims=dims)
        wq_w, scale_w = hidet_b200.symmetric_quantize(wide, quant_type, dims=dims)
        assert torch.equal(_bits(scale), _bits(scale_w)[:cols] if dims == 0 else _bits(scale_w))
        assert torch.equal(wq, wq_w[:, :cols])
        scale = torch.rand(scale.shape, device='cuda', generator=g).to(dtype)
        scale_w = scale if dims == -1 else torch.cat([scale, scale.new_ones(wide.shape[1] - cols)])
        back = hidet_b200.symmetric_dequantize(wq, scale, dims=dims)
        assert torch.equal(_bits(back), _bits(hidet_b200.symmetric_dequantize(wq_w, scale_w, dims=dims)[:, :cols].contiguous()))
