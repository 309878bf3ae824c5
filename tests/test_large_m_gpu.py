"""The kernels for more than a few rows (SM pairs, mid M) at the edges of their tiles, rings and splits."""
import pytest
import torch

import hidet_b200
from hidet_b200 import ffi

pytestmark = pytest.mark.gpu


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


# the kernel on SM pairs, and the mid-M one where columns are few: the heights of tiles, their last rows and columns, k that ends inside a
# stage, one stage, fewer stages than ring slots and more, one tile and several per pair
@pytest.mark.parametrize('m,k,n', [(513, 64, 16), (600, 8, 256), (513, 72, 272), (777, 1000, 528), (1025, 520, 2064), (1500, 2048, 1040), (2048, 1032, 16), (3001, 456, 4112)])
def test_pair_kernel_edges(m, k, n):
    _run(m, k, n, 'KN')
    if k % 16 == 0:
        _run(m, k, n - 8 if n > 16 else n, 'NK')


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=True), dict(bias=True, residual=True), dict(silu=True), dict(silu=True, bias=True, residual=True)])
@pytest.mark.parametrize('m,k,n', [(520, 328, 272), (1100, 136, 4112)])
def test_pair_kernel_epilogues(m, k, n, epilogue):
    _run(m, k, n, 'KN', **epilogue)


# K in one part and in eight, parts of unequal length, tiles of 16 to 128 rows, two row tiles, the last rows and columns
@pytest.mark.parametrize('m,k,n', [(65, 64, 16), (66, 128, 272), (80, 464, 272), (100, 1872, 336), (33, 2736, 10800), (129, 1032, 144), (144, 4096, 528), (24, 4096, 12288), (200, 8200, 1040), (598, 6256, 352)])
def test_mid_kernel_edges(m, k, n):
    _run(m, k, n, 'KN')
    if k % 16 == 0:
        _run(m, k, n - 8 if n > 16 else n, 'NK')


@pytest.mark.parametrize('epilogue', [dict(bias=True), dict(residual=True), dict(silu=True), dict(silu=True, bias=True, residual=True)])
@pytest.mark.parametrize('m,k,n', [(70, 776, 272), (120, 200, 1296)])
def test_mid_kernel_epilogues(m, k, n, epilogue):
    _run(m, k, n, 'KN', **epilogue)


def test_both_kernels_repeat_their_bits():
    for m, k, n in ((100, 3000, 336), (700, 1000, 528)):
        a = torch.randn(m, k, device='cuda').half()
        wq = torch.randint(-128, 128, (k, n), device='cuda', dtype=torch.int8)
        scale = torch.full((n,), 1e-3, device='cuda').half()
        first = hidet_b200.symmetric_quant_matmul(a, wq, scale)
        for _ in range(20):
            assert torch.equal(hidet_b200.symmetric_quant_matmul(a, wq, scale), first)


@pytest.mark.parametrize('ldc,col0,base', [(1284, 0, 0), (1288, 4, 0), (1288, 0, 1)])
def test_outputs_that_16_byte_stores_cannot_write(ldc, col0, base):
    """Refused where only the kernels for many rows serve the call; where the small-M kernel does too, it stores at any element."""
    import ctypes

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
