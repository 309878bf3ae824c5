"""Streams that have only some of the device's SMs (green contexts): no cluster beyond the portable size is launched there."""
import ctypes

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi
from hidet_b200.runtime import workspaces

pytestmark = pytest.mark.gpu


@pytest.fixture
def partial_stream():
    """A stream of a green context of sixteen SMs."""
    driver = pytest.importorskip('cuda.bindings.driver')

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    torch.zeros(1, device='cuda')
    (dev,) = ok(driver.cuDeviceGet(0))
    (sms,) = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    parts, count, _ = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    assert count == 1
    (desc,) = ok(driver.cuDevResourceGenerateDesc([parts[0]], 1))
    (context,) = ok(driver.cuGreenCtxCreate(desc, dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    (stream,) = ok(driver.cuGreenCtxStreamCreate(context, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    ok(driver.cuStreamSynchronize(stream))
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(context))


@pytest.mark.parametrize('m,k,n', [(1, 4096, 1024), (16, 4096, 512), (1, 11008, 4096), (24, 8192, 1024), (1, 256, 688), (4, 65536, 128)])
def test_no_wide_clusters_where_some_sms_are_missing(large_kernels, partial_stream, m, k, n):
    plan = large_kernels.small_plan_on
    plan.argtypes, plan.restype = [ctypes.c_void_p] + [ctypes.c_int64] * 3 + [ctypes.c_void_p], None
    out = (ctypes.c_int * 3)()
    plan(torch.cuda.current_stream().cuda_stream, m, n, k, out)
    whole = out[1]
    plan(partial_stream, m, n, k, out)
    assert out[1] <= 8 and (whole > 8) == (k in (4096, 8192, 11008))
    g = torch.Generator(device='cuda').manual_seed(k)
    a = torch.randn(m, k, generator=g, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n, generator=g, device='cuda') * 1e-3 + 1e-4).half()
    want = (a.double() @ wq.double()) * scale.double()
    got = torch.empty(m, n, dtype=torch.float16, device='cuda')
    ws_ptr, ws_size = workspaces.get(a.device, ffi.func('b200q_qlinear_workspace_bytes')(m, n, k, ffi.LAYOUT_KN))
    torch.cuda.synchronize()
    ffi.func('b200q_qlinear_f16_i8')(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), got.data_ptr(), m, n, k, ffi.LAYOUT_KN, ws_ptr, ws_size, partial_stream)
    torch.cuda.ExternalStream(partial_stream).synchronize()
    # one rounding to f16, and f32 sums of at most 128 steps of 16 k in a row in front of it
    assert float((got.double() - want).abs().max()) <= (2.0 ** -11 + 128 * 2.0 ** -23) * float(want.abs().max())
    assert ffi.func('b200q_check_status')() == ffi.OK
