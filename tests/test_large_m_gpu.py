"""The kernels for more than a few rows (SM pairs, mid M) at the edges of their tiles, rings and splits: first through the public
entry points, where the sizes decide which kernel runs, then each kernel by name with every tile height and split."""
import ctypes

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi

pytestmark = pytest.mark.gpu


SMALL, MID, PAIR = 0, 1, 2


def _plan(large_kernels, m, k, n, silu=False):
    out = (ctypes.c_int * 3)()
    large_kernels.plan(m, n, k, silu, out)
    return out[0]


def _run(m, k, n, layout, bias=False, silu=False, residual=False):
    g = torch.Generator(device='cuda').manual_seed(m * 7 + k + n)
    a = torch.randn(m, k, generator=g, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n) if layout == 'KN' else (n, k), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n, generator=g, device='cuda') * 1e-3 + 1e-4).half()
    more = {}
    if bias:
        more['bias'] = torch.randn(n, generator=g, device='cuda').half()
    if silu:
        more['activation'] = 'silu_mul'
    if residual:
        more['residual'] = torch.randn(m, n // 2 if silu else n, generator=g, device='cuda').half()
    got = hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout=layout, **more)
    assert ffi.func('b200q_check_status')() == ffi.OK
    want = (a.double() @ (wq if layout == 'KN' else wq.t()).double()) * scale.double()
    if bias:
        want += more['bias'].double()
    if silu:
        want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    if residual:
        want += more['residual'].double()
    # one rounding to f16 is half an ulp, 2^-11 of the value; the f32 sums in front of it are far closer
    assert float((got.double() - want).abs().max()) <= 2.0 ** -11 * 1.01 * float(want.abs().max())


# k that ends inside a stage, one stage, fewer stages than ring slots and more, one tile and several per pair of SMs or cluster, the last
# rows and columns
@pytest.mark.parametrize('kind,m,k,n', [(MID, 513, 64, 16), (MID, 600, 8, 256), (MID, 513, 72, 272), (MID, 777, 1000, 528), (PAIR, 1025, 520, 2064), (PAIR, 1500, 2048, 1040),
                                        (MID, 2048, 1032, 16), (PAIR, 3001, 456, 4112), (PAIR, 1000, 4096, 4096), (SMALL, 24, 4096, 12288)])
def test_many_rows(large_kernels, kind, m, k, n):
    assert _plan(large_kernels, m, k, n) == kind
    _run(m, k, n, 'KN')
    if k % 16 == 0:
        _run(m, k, n - 8 if n > 16 else n, 'NK')


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=True), dict(bias=True, residual=True), dict(silu=True), dict(silu=True, bias=True, residual=True)])
@pytest.mark.parametrize('kind,m,k,n', [(MID, 520, 328, 272), (PAIR, 1100, 136, 4112), (PAIR, 1000, 4096, 4096)])
def test_many_rows_with_an_epilogue(large_kernels, kind, m, k, n, epilogue):
    assert _plan(large_kernels, m, k, n, 'silu' in epilogue) == kind
    _run(m, k, n, 'KN', **epilogue)


# K in one part and in eight, parts of unequal length, tiles of 48 to 128 rows, two row tiles, the last rows and columns
@pytest.mark.parametrize('m,k,n', [(65, 64, 16), (66, 128, 272), (80, 464, 272), (100, 1872, 336), (33, 2736, 10800), (129, 1032, 144), (144, 4096, 528), (200, 8200, 1040), (598, 6256, 352)])
def test_a_few_hundred_rows(large_kernels, m, k, n):
    assert _plan(large_kernels, m, k, n) == MID
    _run(m, k, n, 'KN')
    if k % 16 == 0:
        _run(m, k, n - 8 if n > 16 else n, 'NK')


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=True), dict(silu=True), dict(silu=True, bias=True, residual=True)])
@pytest.mark.parametrize('m,k,n', [(70, 776, 272), (120, 200, 1296)])
def test_a_few_hundred_rows_with_an_epilogue(large_kernels, m, k, n, epilogue):
    assert _plan(large_kernels, m, k, n, 'silu' in epilogue) == MID
    _run(m, k, n, 'KN', **epilogue)


def _by_name(lib, kind, tm, cluster, m, k, n, layout='KN', bias=False, silu=False, residual=None, copies=1, lda=0, repeat=1):
    """One call of a kernel with its tiles and split given.  residual: what the length of its rows exceeds the result's by, None without.
    copies > 1: as many destinations, each a column range of wider rows.  lda: the activations are a k range of rows that long."""
    g = torch.Generator(device='cuda').manual_seed(m * 7 + k + n + tm)
    wide = torch.randn(m, lda or k, generator=g, device='cuda').half()
    a = wide[:, 8:8 + k] if lda else wide
    wq = torch.randint(-128, 128, (k, n) if layout == 'KN' else (n, k), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n, generator=g, device='cuda') * 1e-3 + 1e-4).half()
    width = n // 2 if silu else n
    ldc, col0 = (width, 0) if copies == 1 else (width + 40, 24)
    want = (a.double() @ (wq if layout == 'KN' else wq.t()).double()) * scale.double()
    b = torch.randn(n, generator=g, device='cuda').half() if bias else None
    r = torch.randn(m, width + residual, generator=g, device='cuda').half() if residual is not None else None
    if bias:
        want += b.double()
    if silu:
        want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    if r is not None:
        want += r[:, :width].double()
    first = None
    for _ in range(repeat):
        outs = [torch.full((m, ldc), -7.0, dtype=torch.float16, device='cuda') for _ in range(copies)]
        table = (ctypes.c_void_p * copies)(*[o.data_ptr() for o in outs])
        assert lib.launch(kind, tm, cluster, a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, copies, ldc, col0, m, n, k, lda or k, layout == 'NK',
                          b.data_ptr() if bias else None, r.data_ptr() if r is not None else None, width + (residual or 0), silu,
                          torch.cuda.current_stream().cuda_stream) == 0
        if first is None:
            first = outs[0]
            for o in outs:
                # as above; with SiLU the exponential's error, a few units in the last place of f32, is far below that too
                assert float((o[:, col0:col0 + width].double() - want).abs().max()) <= 2.0 ** -11 * 1.01 * float(want.abs().max())
                assert bool((o[:, :col0] == -7.0).all()) and bool((o[:, col0 + width:] == -7.0).all())
        assert torch.equal(outs[0], first)
    assert lib.b200q_check_status() == 0


PAIR_HEIGHTS = [64, 96, 128, 160, 192, 224, 256]   # two accumulators up to 192 rows, one above


@pytest.mark.parametrize('layout', ['KN', 'NK'])
@pytest.mark.parametrize('tm', PAIR_HEIGHTS)
def test_pair_kernel(large_kernels, tm, layout):
    odd = 8 if layout == 'KN' else 16
    # k shorter than a stage, one stage, more stages than any ring holds; a tile of one row, of a whole one and one row, of half of its 32-row
    # blocks; columns of half a CTA's tile, one CTA's of the pair; more tiles than pairs of SMs
    for m, k, n in ((1, odd, 16), (tm + 1, 64, 144), (2 * tm + 33, 1024 + odd, 272), (3 * tm - tm // 2, 192 + odd, 528), (5 * tm + 7, 128 + odd, 4112)):
        _by_name(large_kernels, PAIR, tm, 1, m, k, n if layout == 'KN' else n - 8, layout)


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=0), dict(residual=3), dict(bias=True, residual=8), dict(silu=True), dict(silu=True, bias=True, residual=0),
                                      dict(silu=True, residual=5)])
@pytest.mark.parametrize('tm', PAIR_HEIGHTS)
def test_pair_kernel_epilogues(large_kernels, tm, epilogue):
    for m, k, n in ((2 * tm + 33, 328, 272), (5 * tm + 7, 136, 4112)):
        _by_name(large_kernels, PAIR, tm, 1, m, k, n, **epilogue)


@pytest.mark.parametrize('tm', [128, 192, 224, 256])
def test_pair_kernel_destinations_bands_and_bits(large_kernels, tm):
    _by_name(large_kernels, PAIR, tm, 1, 2 * tm + 33, 520, 1040, copies=3, repeat=3)
    _by_name(large_kernels, PAIR, tm, 1, 2 * tm + 33, 520, 1040, lda=1048)
    _by_name(large_kernels, PAIR, tm, 1, 5 * tm + 40, 1000, 4112, repeat=10)
    # more rows than a band of 48 MB of activations holds, and a last band that is not a whole one
    k = 8192
    band = (48 << 20) // (tm * k * 2)
    _by_name(large_kernels, PAIR, tm, 1, (band + 2) * tm - 9, k, 784, repeat=2)


@pytest.mark.parametrize('layout', ['KN', 'NK'])
@pytest.mark.parametrize('cluster', range(1, 9))
@pytest.mark.parametrize('tm', [16, 48, 64, 80, 112, 128])
def test_mid_kernel(large_kernels, tm, cluster, layout):
    odd = 8 if layout == 'KN' else 16
    # as many stages as CTAs, shares that differ by one, shares beyond every ring; CTAs that own no part of the result; two row tiles
    for m, k, n in ((tm, 64 * cluster, 16), (tm - 5, 64 * (2 * cluster + 1) - odd, 272), (tm + 1, 64 * 9 * cluster + odd, 144)):
        _by_name(large_kernels, MID, tm, cluster, m, k, n if layout == 'KN' else n - 8, layout)


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=0), dict(residual=3), dict(silu=True), dict(silu=True, bias=True, residual=5)])
@pytest.mark.parametrize('tm,cluster', [(32, 1), (64, 3), (96, 8), (128, 5)])
def test_mid_kernel_epilogues(large_kernels, tm, cluster, epilogue):
    _by_name(large_kernels, MID, tm, cluster, 2 * tm - 3, 1096, 336, **epilogue)


@pytest.mark.parametrize('tm,cluster', [(64, 8), (112, 4), (128, 1)])
def test_mid_kernel_destinations_and_bits(large_kernels, tm, cluster):
    _by_name(large_kernels, MID, tm, cluster, 3 * tm - 3, 1096, 336, copies=3, repeat=10)
    _by_name(large_kernels, MID, tm, cluster, tm, 1096, 336, lda=1200)


@pytest.mark.parametrize('kind,m,k,n', [(MID, 100, 3000, 336), (MID, 700, 1000, 528), (PAIR, 1000, 4096, 4096)])
def test_results_repeat_their_bits(large_kernels, kind, m, k, n):
    assert _plan(large_kernels, m, k, n) == kind
    a = torch.randn(m, k, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n), device='cuda', dtype=torch.int8)
    scale = torch.full((n,), 1e-3, device='cuda').half()
    first = hidet_b200.symmetric_quant_matmul(a, wq, scale)
    for _ in range(20):
        assert torch.equal(hidet_b200.symmetric_quant_matmul(a, wq, scale), first)


@pytest.mark.parametrize('ldc,col0,base', [(1284, 0, 0), (1288, 4, 0), (1288, 0, 1)])
def test_outputs_that_16_byte_stores_cannot_write(ldc, col0, base):
    """Refused where only the kernels for many rows serve the call; where the small-M kernel does too, it stores at any element."""
    from hidet_b200.runtime import workspaces

    k, n = 512, 1280
    wq, scale = torch.randint(-128, 128, (k, n), device='cuda', dtype=torch.int8), torch.full((n,), 1e-3, device='cuda').half()
    f, stream = ffi.func('b200q_qlinear_f16_i8_to_peers'), torch.cuda.current_stream().cuda_stream
    for m in (20, 64, 65, 300):
        a = torch.randn(m, k, device='cuda').half()
        out = torch.full((m * ldc + 8,), -7.0, dtype=torch.float16, device='cuda')
        table = (ctypes.c_void_p * 1)(out.data_ptr() + 2 * base)
        ws_ptr, ws_size = workspaces.get(a.device, ffi.func('b200q_qlinear_workspace_bytes')(m, n, k, 0))
        args = (a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, 1, ldc, col0, m, n, k, ws_ptr, ws_size, stream)
        if m > 64:
            with pytest.raises(ffi.BackendException, match='not 16-byte aligned' if base else 'multiples of 8 elements') as e:
                f(*args)
            assert e.value.status == ffi.INVALID_ARGUMENT and bool((out == -7.0).all())
        else:
            f(*args)
            rows = out[base:base + m * ldc].view(m, ldc)
            want = (a.double() @ wq.double()) * scale.double()
            assert float((rows[:, col0:col0 + n].double() - want).abs().max()) <= 2.0 ** -11 * 1.01 * float(want.abs().max())
            assert bool((rows[:, :col0] == -7.0).all()) and bool((rows[:, col0 + n:] == -7.0).all())


# 17 to 24 rows: where one pass of the small-M kernel fills the SMs thinly, in a second wave that is not full, and with long K; and beside those lines
@pytest.mark.parametrize('kind,m,k,n', [(MID, 20, 1024, 32000), (MID, 17, 256, 28688), (MID, 24, 2056, 18432), (MID, 24, 512, 57344), (MID, 18, 520, 65552), (MID, 24, 14336, 4096),
                                        (SMALL, 24, 1024, 12288), (SMALL, 24, 512, 26624), (SMALL, 17, 512, 43008), (SMALL, 24, 1024, 8192), (SMALL, 20, 128, 96000), (SMALL, 24, 14336, 1024)])
def test_17_to_24_rows(large_kernels, kind, m, k, n):
    assert _plan(large_kernels, m, k, n) == kind
    _run(m, k, n, 'KN')
    _run(m, k, n, 'KN', bias=True, silu=True, residual=True)
    if k % 16 == 0:
        _run(m, k, n - 8, 'NK')


# gates at the ends of every range of the epilogue's quotient, in each kernel by name: zeros, where exp(-g) vanishes against 1 and where 1 does
# against it, where it overflows, infinities and NaN
@pytest.mark.parametrize('kind,tm,cluster', [(MID, 48, 1), (MID, 128, 3), (PAIR, 96, 1), (PAIR, 256, 1)])
def test_gates_of_every_magnitude(large_kernels, kind, tm, cluster):
    gates = torch.tensor([0.0, -0.0, 6e-8, -6e-8, 1e-3, -1e-3, 0.5, -0.5, 1.0, -1.0, 9.0, -9.0, 17.0, -17.0, 87.0, -87.0, 88.5, -88.5, 89.0, -89.0, 104.0, -104.0, 6e4, -6e4,
                          float('inf'), float('-inf'), float('nan')])
    m, k, n = tm + 5, 256, 528
    bias = torch.zeros(n)
    bias[0::2] = gates.repeat(n // 2 // len(gates) + 1)[:n // 2]
    bias[1::2] = torch.tensor([1.0, -3.0, 0.25, 1000.0, float('inf')]).repeat(n // 10 + 1)[:n // 2]
    bias = bias.half().cuda()
    a, wq, scale = torch.ones(m, k, dtype=torch.float16, device='cuda'), torch.zeros(k, n, dtype=torch.int8, device='cuda'), torch.ones(n, dtype=torch.float16, device='cuda')
    got = torch.full((m, n // 2), -7.0, dtype=torch.float16, device='cuda')
    table = (ctypes.c_void_p * 1)(got.data_ptr())
    assert large_kernels.launch(kind, tm, cluster, a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, 1, n // 2, 0, m, n, k, k, 0, bias.data_ptr(), None, 0, 1,
                                torch.cuda.current_stream().cuda_stream) == 0
    g, u = bias[0::2].double(), bias[1::2].double()
    want = (g / (1.0 + torch.exp(-g)) * u).half().expand(m, -1)
    keep = ~((g < -88.7) & u.isinf())   # exp overflows in 32 bits there: 0 x inf, which is -inf in 64
    got, want = got[:, keep], want[:, keep]
    assert torch.equal(got.isnan(), want.isnan())
    finite = want.isfinite()
    assert torch.equal(got[~finite & ~want.isnan()], want[~finite & ~want.isnan()])
    # f32 in front of one rounding to f16: an ulp of the value at most, or of the smallest number; exp's own error is 2^-20 of it at 104
    err = (got.double() - want.double()).abs()[finite]
    assert bool((err <= 2.0 ** -10 * want.double().abs()[finite] + 2.0 ** -24).all())
    assert large_kernels.b200q_check_status() == 0
