"""CudaGraph: who owns the scratch that a captured sequence of launches writes to."""
import gc

import pytest
import torch

import hidet_b200
from hidet_b200 import ffi

pytestmark = pytest.mark.gpu


def _problem(m, k, n, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    wq, scale = hidet_b200.symmetric_quantize(torch.randn(k, n, device='cuda', generator=gen).half() * 0.02, 'int8', dims=0)
    return torch.randn(m, k, device='cuda', generator=gen).half(), wq, scale


def _graph(a, wq, scale):
    return hidet_b200.CudaGraph(lambda: [a.clone()], lambda inputs: [hidet_b200.symmetric_quant_matmul(inputs[0], wq, scale)])


def test_graphs_on_one_pooled_stream_and_eager_calls_between_their_replays():
    """Streams come from a small pool: later graphs capture on the stream of earlier ones, whose scratch must stay theirs, and
    eager calls there grow a scratch of their own."""
    small, larger = _problem(4, 16384, 256, 1), _problem(16, 16384, 1024, 2)
    workspace = ffi.func('b200q_qlinear_workspace_bytes')
    assert 0 < workspace(4, 256, 16384, ffi.LAYOUT_KN) < workspace(16, 1024, 16384, ffi.LAYOUT_KN)
    want = [hidet_b200.symmetric_quant_matmul(*p) for p in (small, larger)]
    graphs, streams = [], []
    while len(streams) == len(set(streams)):
        assert len(graphs) < 200
        graphs.append(_graph(*small))
        streams.append(graphs[-1]._stream.cuda_stream)
    first = streams.index(streams[-1])
    pair = [graphs[first], graphs[-1]]
    assert pair[0]._scratch.data_ptr() != pair[1]._scratch.data_ptr()
    graphs.append(_graph(*larger))
    stream = pair[0]._stream
    with torch.cuda.stream(stream):
        for _ in range(5):
            for g in pair:
                g.run_async([small[0]], stream)
                assert torch.equal(g.outputs[0], want[0])
                eager = [hidet_b200.symmetric_quant_matmul(*p) for p in (small, larger)]
                assert torch.equal(eager[0], want[0]) and torch.equal(eager[1], want[1])
    assert torch.equal(graphs[-1].run([larger[0]])[0], want[1])
    assert ffi.func('b200q_check_status')() == ffi.OK


def test_scratch_of_a_dropped_graph_outlives_its_replays():
    a, wq, scale = _problem(4, 16384, 256, 3)
    graph = _graph(a, wq, scale)
    want = graph.run([a])[0].clone()
    scratch, size, stream = graph._scratch.data_ptr(), graph._scratch.numel(), graph._stream
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(400_000_000)  # the replay stays in flight for a while
        got = graph.run_async([a], other)[0]
        done = torch.cuda.Event()
        done.record()
    del graph
    gc.collect()
    with torch.cuda.stream(stream):
        taken = [torch.empty(size, dtype=torch.uint8, device='cuda') for _ in range(16)]
    assert not done.query(), 'the replay is over too early for this test to show anything'
    assert not any(t.data_ptr() < scratch + size and scratch < t.data_ptr() + size for t in taken)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
