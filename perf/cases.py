"""Workloads of the weight-only quantized linear path, as programs that use this package run it.

listed() names a fixed set, draw() gives further ones of the same ranges; prepare() makes what a program holds
before the call, run() is one pass through the public entry points, work() the bytes and operations a pass cannot do
without and tolerance() how far another correct implementation may be from it.

Kinds of case:
    linear      one eager call of symmetric_quant_matmul (KN: the package's own weight layout; NK: torch.nn.Linear's)
    step        one decode step: a CUDA graph over the embedding lookup, `layers` decoder blocks' linears with their fused
                epilogues and the output projection, replayed for a batch of m token ids
    quantize    symmetric_quantize of one weight, as done when a model is loaded or rewritten
    dequantize  symmetric_dequantize of one weight
    w4          one call of a w4a16 linear (4-bit codes, group scales, zero points)
"""
import math

import torch

import hidet_b200
from hidet_b200.quant import cast_f16_to_u4, interleave_gate_up, w4a16_linear

DTYPES = {'float16': torch.float16, 'bfloat16': torch.bfloat16, 'float32': torch.float32}
LARGEST_FLOPS = 2.0 * 2048 * 8192 * 28672


def listed():
    return [
        # The smallest call: one token through a narrow projection (the small decoder configuration's hidden -> FFN).
        # Launch and host time.
        dict(name='linear_1x256x688', kind='linear', m=1, k=256, n=688, layout='KN', epilogue='none'),
        # Batch-1 decoding at 7B widths: what a generation loop replays per token.  Streaming the weights.
        dict(name='step_b1', kind='step', m=1, hidden=4096, ffn=11008, layers=4, vocab=32000),
        # The same step for sixteen sequences decoded together.
        dict(name='step_b16', kind='step', m=16, hidden=4096, ffn=11008, layers=4, vocab=32000),
        # Output projection over a vocabulary with two added tokens: rows of the weight are not multiples of 16 bytes.
        dict(name='linear_7x4096x32002', kind='linear', m=7, k=4096, n=32002, layout='KN', epilogue='none'),
        # Larger decode batch / short prompt on a weight kept as torch.nn.Linear stores it.
        dict(name='linear_64x4096x11008_nk', kind='linear', m=64, k=4096, n=11008, layout='NK', epilogue='none'),
        # A 512-token prompt through the fused gate + up projection (SiLU and product inside the kernel).
        dict(name='linear_512x4096x22016_silu', kind='linear', m=512, k=4096, n=22016, layout='KN', epilogue='silu_mul'),
        # The largest: 2048 prompt rows through a 70B-shaped FFN projection.  Tensor cores.
        dict(name='linear_2048x8192x28672', kind='linear', m=2048, k=8192, n=28672, layout='KN', epilogue='none'),
        # Quantizing an FFN weight per output channel, in the package's own layout.
        dict(name='quantize_f16_cols', kind='quantize', rows=4096, cols=11008, dtype='float16', quant='int8', dims=0),
        # Quantizing a torch.nn.Linear weight of a bfloat16 checkpoint per output row.
        dict(name='quantize_bf16_rows', kind='quantize', rows=11008, cols=4096, dtype='bfloat16', quant='int8', dims=-1),
        # Restoring a weight (an operator outside the quantized path wants it back).
        dict(name='dequantize_f16_cols', kind='dequantize', rows=4096, cols=11008, dtype='float16', quant='int8', dims=0),
        # 4-bit decoding, one sequence ...
        dict(name='w4_1x4096x12288', kind='w4', m=1, k=4096, n=12288, group=128, zeros=True),
        # ... and a batch of sixteen.
        dict(name='w4_16x12288x4096', kind='w4', m=16, k=12288, n=4096, group=128, zeros=True),
    ]


def _log(rng, low, high, multiple=1):
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(['linear'] * 6 + ['step'] * 2 + ['quantize'] * 2 + ['dequantize'] + ['w4'] * 2)
    if kind == 'linear':
        if rng.random() < 1 / 6:  # rows that are not multiples of 16 bytes: vocabularies with added tokens, odd feature counts
            return dict(kind=kind, m=_log(rng, 1, 16), k=_log(rng, 256, 8192, 8), n=_log(rng, 256, 32768, 16) + rng.choice([2, 4, 6, 8, 10]),
                        layout='KN', epilogue='none')
        layout = rng.choice(['KN', 'KN', 'NK'])
        epilogue = 'none' if layout == 'NK' else rng.choice(['none', 'none', 'bias', 'residual', 'silu_mul'])
        while True:
            c = dict(kind=kind, m=_log(rng, 1, 2048), k=_log(rng, 256, 11008, 16), n=_log(rng, 256, 28672, 16), layout=layout, epilogue=epilogue)
            if 2.0 * c['m'] * c['k'] * c['n'] <= LARGEST_FLOPS:
                return c
    if kind == 'step':
        hidden = _log(rng, 1024, 5120, 128)
        return dict(kind=kind, m=_log(rng, 1, 32), hidden=hidden, ffn=int(hidden * rng.uniform(2.5, 4.0)) // 16 * 16, layers=rng.randint(1, 4),
                    vocab=_log(rng, 1000, 32000, 16))
    if kind in ('quantize', 'dequantize'):
        rows, cols = _log(rng, 256, 12288, 1), _log(rng, 256, 12288, rng.choice([1, 8, 16, 16]))
        return dict(kind=kind, rows=rows, cols=cols, dtype=rng.choice(['float16', 'float16', 'bfloat16', 'float32']),
                    quant=rng.choice(['int8', 'int8', 'int8', 'int16']), dims=rng.choice([0, -1]))
    group = rng.choice([32, 64, 128, 128, 256])
    return dict(kind=kind, m=_log(rng, 1, 64), k=_log(rng, 512, 12288, group), n=_log(rng, 256, 12288, 8), group=group, zeros=rng.random() < 0.7)


def _normal(gen, shape, std, dtype=torch.float16):
    return torch.randn(shape, generator=gen, device='cuda', dtype=torch.float32).mul_(std).to(dtype)


def _decode_step(case, gen):
    m, hidden, ffn, layers, vocab = (case[key] for key in ('m', 'hidden', 'ffn', 'layers', 'vocab'))

    def weight(k, n):
        return hidet_b200.symmetric_quantize(_normal(gen, (k, n), 0.6 / math.sqrt(k)), 'int8', dims=0)

    table = hidet_b200.symmetric_quantize(_normal(gen, (vocab, hidden), 1.0), 'int8', dims=-1)
    blocks = []
    for _ in range(layers):
        qkv, out, down = weight(hidden, 3 * hidden), weight(hidden, hidden), weight(ffn, hidden)
        gate, up = weight(hidden, ffn), weight(hidden, ffn)
        blocks.append((qkv, out, tuple(interleave_gate_up(g, u) for g, u in zip(gate, up)), down))
        del gate, up
    head = weight(hidden, vocab)
    attention = _normal(gen, (layers, m, hidden), 1.0)  # what attention (not part of this package) hands to the output projections
    ids = torch.randint(0, vocab, (m,), generator=gen, device='cuda')

    def step(inputs):
        linear = hidet_b200.symmetric_quant_matmul
        x = hidet_b200.symmetric_dequantize_take(*table, inputs[0])
        outputs = []
        for i, (qkv, out, gate_up, down) in enumerate(blocks):
            outputs.append(linear(x, *qkv))
            x = linear(attention[i], *out, residual=x)
            x = linear(linear(x, *gate_up, activation='silu_mul'), *down, residual=x)
        outputs.append(linear(x, *head))
        return outputs

    graph = hidet_b200.CudaGraph(lambda: [torch.zeros_like(ids)], step, ref_objs=[table, blocks, head, attention])
    return {'kind': 'step', 'graph': graph, 'ids': ids}


def prepare(case, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    kind = case['kind']
    if kind == 'step':
        return _decode_step(case, gen)
    if kind == 'linear':
        m, k, n = case['m'], case['k'], case['n']
        w = _normal(gen, (k, n) if case['layout'] == 'KN' else (n, k), 0.02)
        wq, scale = hidet_b200.symmetric_quantize(w, 'int8', dims=0 if case['layout'] == 'KN' else -1)
        more = {}
        if case['epilogue'] == 'bias':
            more['bias'] = _normal(gen, (n,), 0.5)
        elif case['epilogue'] == 'residual':
            more['residual'] = _normal(gen, (m, n), 1.0)
        elif case['epilogue'] == 'silu_mul':
            more['activation'] = 'silu_mul'
        return {'kind': kind, 'a': _normal(gen, (m, k), 1.0), 'wq': wq, 'scale': scale, 'layout': case['layout'], 'more': more}
    if kind in ('quantize', 'dequantize'):
        w = _normal(gen, (case['rows'], case['cols']), 0.02, DTYPES[case['dtype']])
        state = {'kind': kind, 'quant': case['quant'], 'dims': case['dims']}
        if kind == 'quantize':
            return dict(state, w=w)
        wq, scale = hidet_b200.symmetric_quantize(w, case['quant'], dims=case['dims'])
        return dict(state, wq=wq, scale=scale)
    m, k, n, group = case['m'], case['k'], case['n'], case['group']
    codes = cast_f16_to_u4(torch.randint(0, 16, (k, n), generator=gen, device='cuda').to(torch.float16))
    scale = torch.rand((k // group, n), generator=gen, device='cuda').mul_(0.01).add_(0.002).to(torch.float16)
    zeros = torch.rand((k // group, n), generator=gen, device='cuda').mul_(15).to(torch.float16) if case['zeros'] else None
    linear = w4a16_linear('w4', k, n, group, with_zp=case['zeros'])
    return {'kind': kind, 'linear': linear, 'a': _normal(gen, (m, k), 1.0), 'codes': codes, 'scale': scale, 'zeros': zeros}


def run(state):
    kind = state['kind']
    if kind == 'linear':
        return hidet_b200.symmetric_quant_matmul(state['a'], state['wq'], state['scale'], weight_layout=state['layout'], **state['more'])
    if kind == 'step':
        return state['graph'].run_async([state['ids']])
    if kind == 'quantize':
        return hidet_b200.symmetric_quantize(state['w'], state['quant'], dims=state['dims'])
    if kind == 'dequantize':
        return hidet_b200.symmetric_dequantize(state['wq'], state['scale'], dims=state['dims'])
    return state['linear'](state['a'], state['codes'], state['scale'], state['zeros'])


def work(case):
    kind = case['kind']
    if kind == 'linear':
        m, k, n = case['m'], case['k'], case['n']
        bytes_ = k * n + 2 * m * k + 2 * n + (m * n if case['epilogue'] == 'silu_mul' else 2 * m * n)
        bytes_ += 2 * n if case['epilogue'] == 'bias' else 2 * m * n if case['epilogue'] == 'residual' else 0
        return {'bytes': bytes_, 'flops': 2.0 * m * k * n}
    if kind == 'step':
        m, h, f, layers, vocab = (case[key] for key in ('m', 'hidden', 'ffn', 'layers', 'vocab'))
        weights = layers * (4 * h * h + 3 * h * f) + h * vocab
        scales = layers * (3 * h + h + 2 * f + h) + vocab
        # rows that enter or leave a step: table rows and ids, attention results, q / k / v and logits
        rows = h + 2 + 8 + layers * (2 * h + 2 * 3 * h) + 2 * vocab
        return {'bytes': weights + 2 * scales + m * rows, 'flops': 2.0 * m * weights}
    if kind in ('quantize', 'dequantize'):
        size, q = DTYPES[case['dtype']].itemsize, 1 if case['quant'] == 'int8' else 2
        return {'bytes': case['rows'] * case['cols'] * (size + q) + size * (case['cols'] if case['dims'] == 0 else case['rows']),
                'flops': 2.0 * case['rows'] * case['cols']}
    m, k, n = case['m'], case['k'], case['n']
    groups = k // case['group']
    return {'bytes': k * n // 2 + 2 * groups * n * (2 if case['zeros'] else 1) + 2 * m * k + 2 * m * n, 'flops': 2.0 * m * k * n}


def tolerance(case):
    if case['kind'] in ('quantize', 'dequantize'):
        return 'exact'  # codes, scales and restored values are defined to the bit
    if case['kind'] == 'step':
        return {'rel': 2e-3, 'max': 2e-2}  # float16 roundings between up to nineteen dependent launches
    return {'rel': 1e-3, 'max': 4e-3}  # float32 sums, one rounding to float16 (half an ulp is 4.9e-4 of the value)
