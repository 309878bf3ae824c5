"""The one-SM kernel for many rows and its split over K, which the library runs for the multicast delivery only: here on ordinary
destinations, one and several, whole and as column ranges of wider rows."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

HEAD = 65536 * 4   # the split leaves the head of the workspace alone


# rows of 256- and 64-row tiles and their last ones, k that ends inside a stage, columns that end inside a tile; then the shapes
# whose K is split, an eight-way column shard of the 70B layer first
@pytest.mark.parametrize('m,k,n,split', [(33, 72, 16, False), (65, 64, 144, False), (300, 520, 4112, False), (2048, 520, 10800, False), (700, 4096, 8192, False),
                                         (256, 8192, 3584, True), (300, 4096, 1024, True), (65, 2048, 144, True), (100, 8200, 528, True)])
@pytest.mark.parametrize('scale_offset', [0, 1])
def test_one_sm_kernel(large_kernels, m, k, n, split, scale_offset):
    g = torch.Generator(device='cuda').manual_seed(m + k + n)
    a = torch.randn(m, k, generator=g, device='cuda').half()
    wq = torch.randint(-128, 128, (k, n), generator=g, device='cuda', dtype=torch.int8)
    scale = (torch.rand(n + 1, generator=g, device='cuda') * 1e-3 + 1e-4).half()[scale_offset:scale_offset + n]
    ldc, col0, count = n + 40, 24, 2
    want = (a.double() @ wq.double()) * scale.double()
    room = torch.zeros(HEAD + (8 << 20) * 16, dtype=torch.uint8, device='cuda')
    room[HEAD:] = 255   # NaN as f32: what is not written must not be read
    runs = []
    for size in [room.numel(), room.numel()] + ([0] if split else []):   # without scratch: the same sums in one part
        dsts = [torch.full((m, ldc), -7.0, dtype=torch.float16, device='cuda') for _ in range(count)]
        table = (ctypes.c_void_p * count)(*[d.data_ptr() for d in dsts])
        parts = large_kernels.launch_one_sm(a.data_ptr(), wq.data_ptr(), scale.data_ptr(), table, count, ldc, col0, m, n, k, room.data_ptr() if size else None, size,
                                            torch.cuda.current_stream().cuda_stream)
        assert parts > 1 if split and size else parts == 1
        for d in dsts:
            # one rounding to f16 is half an ulp, 2^-11 of the value; the f32 sums in front of it are far closer
            assert float((d[:, col0:col0 + n].double() - want).abs().max()) <= 2.0 ** -11 * 1.01 * float(want.abs().max())
            assert bool((d[:, :col0] == -7.0).all()) and bool((d[:, col0 + n:] == -7.0).all())
        runs.append(dsts[0])
    assert torch.equal(runs[0], runs[1]) and not bool(room[:HEAD].any())
    assert large_kernels.b200q_check_status() == 0
