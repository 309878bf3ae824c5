"""The small-M kernel's splits that meet in the workspace: deep and narrow weights, whose clusters are several to an output tile."""
import ctypes

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi
from hidet_b200.runtime import workspaces

pytestmark = pytest.mark.gpu


def _groups(large_kernels, m, k, n):
    out = (ctypes.c_int * 3)()
    large_kernels.small_plan(m, n, k, out)
    return out[2]


def _operands(m, k, n, layout='KN', seed=0):
    g = torch.Generator(device='cuda').manual_seed(m + k + n + seed)
    a = torch.randn(m, k, generator=g, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n) if layout == 'KN' else (n, k), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n, generator=g, device='cuda') * 1e-3 + 1e-4).half()
    return a, wq, scale, (a.double() @ (wq if layout == 'KN' else wq.t()).double()) * scale.double()


def _close(got, want, k):
    # one rounding to f16, half an ulp of the value; in front of it f32 sums, an ulp of the partial sum for each 16 k of a split, which is at
    # most a hundred-and-twenty-eighth of K here, and a few for the partials
    assert float((got.double() - want).abs().max()) <= (2.0 ** -11 + (k / 128 / 16 + 16) * 2.0 ** -23) * float(want.abs().max())


SHAPES = [(32768, 16), (32776, 256), (40968, 1024), (65536, 128), (65528, 144), (131072, 64)]


# rows of every form of the kernel and of two row blocks; k that ends inside a step, splits with fewer steps than others or none; the last columns
@pytest.mark.parametrize('m', [1, 2, 4, 5, 8, 9, 16, 17, 24])
@pytest.mark.parametrize('k,n', SHAPES)
def test_splits_through_the_workspace(large_kernels, m, k, n):
    if m <= 16 or n * k <= 6 * 1024 * 1024 or k >= 65528:
        assert _groups(large_kernels, m, k, n) > 1
    a, wq, scale, want = _operands(m, k, n)
    got = hidet_b200.symmetric_quant_matmul(a, wq, scale)
    _close(got, want, k)
    assert torch.equal(hidet_b200.symmetric_quant_matmul(a, wq, scale), got)   # one order of the sums, counters that are zero again
    if k % 16 == 0:
        a, wq, scale, want = _operands(m, k, n - 7, 'NK')
        _close(hidet_b200.symmetric_quant_matmul(a, wq, scale, weight_layout='NK'), want, k)
    assert ffi.func('b200q_check_status')() == ffi.OK


@pytest.mark.parametrize('m', [1, 4, 7, 16, 24])
@pytest.mark.parametrize('bias,act,residual', [(True, None, False), (False, None, True), (False, 'silu_mul', False), (True, 'silu_mul', True)])
def test_epilogues_behind_the_workspace(large_kernels, m, bias, act, residual):
    k, n = 65536, 144
    assert _groups(large_kernels, m, k, n) > 1
    a, wq, scale, _ = _operands(m, k, n)
    scale = scale / 64   # gates of ordinary size
    want = (a.double() @ wq.double()) * scale.double()
    more = {}
    if bias:
        more['bias'] = torch.randn(n, device='cuda').half()
        want = want + more['bias'].double()
    if act:
        more['activation'] = act
        want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    if residual:
        more['residual'] = torch.randn(m, want.shape[1], device='cuda').half()
        want = want + more['residual'].double()
    _close(hidet_b200.symmetric_quant_matmul(a, wq, scale, **more), want, k)


@pytest.mark.parametrize('m', [1, 16])
def test_workspace_is_left_as_it_was_asked_for_and_refused_when_short(large_kernels, m):
    k, n = 40960, 256
    assert _groups(large_kernels, m, k, n) > 1
    a, wq, scale, want = _operands(m, k, n)
    need = ffi.func('b200q_qlinear_workspace_bytes')(m, n, k, ffi.LAYOUT_KN)
    counters = 65536 * 4   # its head
    assert need > counters
    stream = torch.cuda.current_stream().cuda_stream
    space = torch.zeros(need + 4096, dtype=torch.uint8, device='cuda')
    space[need:] = 0x5a
    out = torch.full((m, n), -7.0, dtype=torch.float16, device='cuda')
    call = ffi.func('b200q_qlinear_f16_i8')
    with pytest.raises(ffi.BackendException, match='workspace'):
        call(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), out.data_ptr(), m, n, k, ffi.LAYOUT_KN, space.data_ptr(), need - 1, stream)
    call(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), out.data_ptr(), m, n, k, ffi.LAYOUT_KN, space.data_ptr(), need, stream)
    _close(out, want, k)
    assert not space[:counters].any() and space[counters:need].any() and bool((space[need:] == 0x5a).all())
    static = torch.empty_like(out)
    ffi.func('b200q_qlinear_f16_i8_static')(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), static.data_ptr(), m, n, k, ffi.LAYOUT_KN, stream)
    assert torch.equal(static, out)


def test_destinations_behind_the_workspace(large_kernels):
    m, k, n, ldc, col0 = 7, 40960, 272, 301, 13
    assert _groups(large_kernels, m, k, n) > 1
    a, wq, scale, want = _operands(m, k, n)
    outs = [torch.full((m, ldc), -7.0, dtype=torch.float16, device='cuda') for _ in range(2)]
    table = (ctypes.c_void_p * 2)(*[o.data_ptr() for o in outs])
    need = ffi.func('b200q_qlinear_workspace_bytes')(m, n, k, ffi.LAYOUT_KN)
    ws_ptr, ws_size = workspaces.get(a.device, need)
    ffi.func('b200q_qlinear_f16_i8_to_peers')(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, 2, ldc, col0, m, n, k, ws_ptr, ws_size,
                                             torch.cuda.current_stream().cuda_stream)
    for o in outs:
        _close(o[:, col0:col0 + n], want, k)
        assert bool((o[:, :col0] == -7.0).all()) and bool((o[:, col0 + n:] == -7.0).all())


def _graph(a, wq, scale):
    return hidet_b200.CudaGraph(lambda: [a.clone()], lambda inputs: [hidet_b200.symmetric_quant_matmul(inputs[0], wq, scale)])


def test_graphs_and_eager_calls_that_write_scratch_on_one_stream(large_kernels):
    """Graphs captured on one pooled stream keep scratch of their own; eager calls there, of a smaller and a larger need, have theirs."""
    problems = [_operands(4, 40960, 256, seed=1)[:3], _operands(16, 65536, 512, seed=2)[:3]]
    for a, wq, _ in problems:
        assert _groups(large_kernels, a.shape[0], *wq.shape) > 1
    want = [hidet_b200.symmetric_quant_matmul(*p) for p in problems]
    graphs = [_graph(*p) for p in problems for _ in range(2)]
    stream = graphs[0]._stream
    with torch.cuda.stream(stream):
        for _ in range(5):
            for i, g in enumerate(graphs):
                got = g.run_async([problems[i // 2][0]], stream)[0]
                eager = [hidet_b200.symmetric_quant_matmul(*p) for p in problems]
                assert torch.equal(got, want[i // 2]) and torch.equal(eager[0], want[0]) and torch.equal(eager[1], want[1])
    assert ffi.func('b200q_check_status')() == ffi.OK


def test_streams_that_write_scratch_at_the_same_time(large_kernels):
    p = _operands(8, 65536, 512)[:3]
    assert _groups(large_kernels, 8, 65536, 512) > 1
    want = hidet_b200.symmetric_quant_matmul(*p)
    streams = [torch.cuda.Stream() for _ in range(4)]
    got = [[] for _ in streams]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, results in zip(streams, got):
            with torch.cuda.stream(s):
                results.append(hidet_b200.symmetric_quant_matmul(*p))
    torch.cuda.synchronize()
    assert all(torch.equal(r, want) for results in got for r in results)


@pytest.mark.parametrize('m', [17, 24])
def test_codes_of_17_rows_and_more_may_be_late_there_too(large_kernels, nvcc_library, m):
    k, n = 65536, 128
    assert _groups(large_kernels, m, k, n) > 1
    copy = nvcc_library('late_copy.cu').late_copy
    copy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    a, first, scale, _ = _operands(m, k, n)
    weights = [first, -1 - first]   # no two codes alike
    want = [hidet_b200.symmetric_quant_matmul(a, w, scale) for w in weights]
    buffer = torch.zeros_like(first)
    for i in range(6):
        assert copy(buffer.data_ptr(), weights[i % 2].data_ptr(), buffer.numel() // 4, 40000, torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(hidet_b200.symmetric_quant_matmul(a, buffer, scale), want[i % 2])
