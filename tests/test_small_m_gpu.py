"""The small-M kernel: its last step (four columns a thread, counts and addresses that are not multiples of four) and its splits."""
import ctypes

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi
from hidet_b200.runtime import workspaces

pytestmark = pytest.mark.gpu


def _operands(m, k, n, layout):
    g = torch.Generator(device='cuda').manual_seed(m + k + n)
    a = torch.randn(m, k, generator=g, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n) if layout == 'KN' else (n, k), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n, generator=g, device='cuda') * 1e-3 + 1e-4).half()
    want = (a.double() @ (wq if layout == 'KN' else wq.t()).double()) * scale.double()
    return a, wq, scale, want


def _close(got, want):
    # one rounding to f16, half an ulp of the value; the f32 sums in front of it are far closer
    assert float((got.double() - want).abs().max()) <= 2.0 ** -11 * 1.01 * float(want.abs().max())


@pytest.mark.parametrize('m', [1, 2, 3, 5, 6, 7, 8, 9, 16])
@pytest.mark.parametrize('k,n', [(1024, 129), (2048, 258), (4096, 1027), (512, 4095)])
def test_odd_column_counts(m, k, n):
    a, wq, scale, want = _operands(m, k, n, 'NK')
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout='NK'), want)


@pytest.mark.parametrize('m', [1, 7, 16])
@pytest.mark.parametrize('ldc,col0', [(1293, 7), (1290, 2), (1284, 4)])
def test_destinations_at_any_element(m, ldc, col0):
    a, wq, scale, want = _operands(m, 1536, 1280, 'KN')
    out = torch.full((m, ldc), -7.0, dtype=torch.float16, device='cuda')
    table = (ctypes.c_void_p * 1)(out.data_ptr())
    ws_ptr, ws_size = workspaces.get(a.device, ffi.func('b200q_qlinear_workspace_bytes')(m, 1280, 1536, 0))
    ffi.func('b200q_qlinear_f16_i8_to_peers')(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, 1, ldc, col0, m, 1280, 1536, ws_ptr, ws_size,
                                             torch.cuda.current_stream().cuda_stream)
    _close(out[:, col0:col0 + 1280], want)
    assert bool((out[:, :col0] == -7.0).all()) and bool((out[:, col0 + 1280:] == -7.0).all())


# scales, bias and residual at any element, rows of the residual and of the result of any length
@pytest.mark.parametrize('m', [1, 4, 5, 8, 16])
@pytest.mark.parametrize('offset,ldr', [(0, 1280), (1, 1283), (2, 1281), (3, 1286), (4, 1284)])
@pytest.mark.parametrize('k', [256, 1536])   # one CTA a tile; K split
def test_operands_of_the_epilogue_at_any_element(m, k, offset, ldr):
    n = 1280
    a, wq, scale, want = _operands(m, k, n, 'KN')

    def at_offset(t):
        out = torch.empty(offset + t.numel(), dtype=torch.float16, device='cuda')
        out[offset:] = t.flatten()
        return out, out.data_ptr() + 2 * offset

    bias, residual = torch.randn(n, device='cuda').half(), torch.randn(m, ldr, device='cuda').half()
    keep = [at_offset(t) for t in (scale, bias, residual)]
    out = torch.empty(m, n, dtype=torch.float16, device='cuda')
    ws_ptr, ws_size = workspaces.get(a.device, ffi.func('b200q_qlinear_workspace_bytes')(m, n, k, 0))
    ep = ffi.Epilogue(keep[1][1], keep[2][1], ldr, 0)
    ffi.func('b200q_qlinear_f16_i8_fused')(a.data_ptr(), wq.data_ptr(), keep[0][1], out.data_ptr(), m, n, k, 0, ctypes.byref(ep), ws_ptr, ws_size,
                                          torch.cuda.current_stream().cuda_stream)
    _close(out, want + bias.double() + residual[:, :n].double())


def _plan(large_kernels, m, k, n):
    out = (ctypes.c_int * 3)()
    large_kernels.small_plan(m, n, k, out)
    return tuple(out)


# clusters beyond eight CTAs: nine to sixteen with slices of every width, splits that get fewer steps than others or none, a last step that is
# cut short, tiles that are; short K in two to four splits
@pytest.mark.parametrize('m', [1, 2, 3, 8, 9, 16, 17, 24])
@pytest.mark.parametrize('k,n', [(3072, 16), (3080, 272), (4096, 1024), (4104, 16), (11008, 4096), (11024, 3328), (12288, 4592), (16376, 512), (9000, 5120)])
def test_wide_clusters(large_kernels, m, k, n):
    assert _plan(large_kernels, m, k, n)[1] > 8 or m > 16 or (m > 8 and n > 1536)
    a, wq, scale, want = _operands(m, k, n, 'KN')
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale), want)
    if k % 16 == 0:
        a, wq, scale, want = _operands(m, k, n + 1, 'NK')
        _close(hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout='NK'), want)


@pytest.mark.parametrize('m', [1, 4, 7, 16])
@pytest.mark.parametrize('k,n,splits', [(192, 272, 1), (200, 272, 2), (256, 688, 2), (328, 2048, 3), (512, 16, 4), (1016, 1040, 4), (256, 12288, 2), (512, 16384, 2)])
def test_short_splits(large_kernels, m, k, n, splits):
    assert _plan(large_kernels, m, k, n)[1] == splits
    a, wq, scale, want = _operands(m, k, n, 'KN')
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale), want)


@pytest.mark.parametrize('m', [17, 20, 23, 24, 25])
@pytest.mark.parametrize('k,n', [(4096, 1536), (1000, 6304), (2048, 3072), (6264, 1024), (520, 16400)])
def test_rows_up_to_24_in_one_pass(large_kernels, m, k, n):
    if k * n >= 6 * 1024 * 1024:
        assert (_plan(large_kernels, m, k, n)[0] == m) == (m <= 24)
    a, wq, scale, want = _operands(m, k, n, 'KN')
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale), want)
    gate = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    residual = torch.randn(m, n // 2, device='cuda').half()
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale, activation='silu_mul', residual=residual), gate + residual.double())


# every form in every cluster size that the plan may take, by name: slices of every width, ranks that own no columns, splits that get fewer steps
# than others or none, rows short of the form's, the last columns
@pytest.mark.parametrize('cluster', [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 16])
@pytest.mark.parametrize('form,rows', [(0, [1, 2, 4]), (1, [3, 5, 8]), (2, [9, 16, 31]), (3, [17, 20, 24])])
def test_every_cluster(large_kernels, cluster, form, rows):
    p, i, n = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
    launch = large_kernels.launch_small
    launch.argtypes = [i, i, p, p, p, p, n, n, n, i, p, p, i, p]
    stream = torch.cuda.current_stream().cuda_stream
    for m in rows:
        for k, cols, layout in ((3080, 272, 'KN'), (512, 16, 'KN'), (1040, 391, 'NK')):
            a, wq, scale, want = _operands(m, k, cols, layout)
            out = torch.full((m, cols), -7.0, dtype=torch.float16, device='cuda')
            assert launch(form, cluster, a.data_ptr(), wq.data_ptr(), scale.data_ptr(), out.data_ptr(), m, cols, k, layout == 'NK', None, None, 0, stream) == 0
            _close(out, want)
            if cols % 2 == 0:
                bias, residual = torch.randn(cols, device='cuda').half(), torch.randn(m, cols // 2, device='cuda').half()
                out = torch.full((m, cols // 2), -7.0, dtype=torch.float16, device='cuda')
                assert launch(form, cluster, a.data_ptr(), wq.data_ptr(), scale.data_ptr(), out.data_ptr(), m, cols, k, 0, bias.data_ptr(), residual.data_ptr(), 1, stream) == 0
                y = want + bias.double()
                _close(out, torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2] + residual.double())
    assert large_kernels.b200q_check_status() == 0


def test_no_clusters_of_fifteen(large_kernels):
    """Slices of twelve columns from fifteen CTAs would not fit where they are received."""
    p, i, n = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
    launch = large_kernels.launch_small
    launch.argtypes = [i, i, p, p, p, p, n, n, n, i, p, p, i, p]
    a, wq, scale, _ = _operands(4, 3072, 256, 'KN')
    out = torch.empty(4, 256, dtype=torch.float16, device='cuda')
    for cluster in (15, 17):
        assert launch(0, cluster, a.data_ptr(), wq.data_ptr(), scale.data_ptr(), out.data_ptr(), 4, 256, 3072, 0, None, None, 0, torch.cuda.current_stream().cuda_stream) == ffi.INVALID_ARGUMENT
