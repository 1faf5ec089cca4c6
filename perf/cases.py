"""The workloads this library is timed on: what a program that uses its operators asks of it.

``listed()`` names the fixed cases, ``draw(rng)`` gives one more of the same ranges.  A case is a dict
of plain values whose ``kind`` says which operator (or chain of operators) it runs:

* ``network``  the 53 int8 convolutions of ResNet-50 (the shapes of ``unit_b200.resnet50``) on ``n``
               images: the 7x7 stem, then sixteen bottleneck blocks in which every convolution reads
               its predecessor's u8 NCHW16c output and the expanding one adds the block's input.  The
               program plans every layer once and runs the plans, one after the other (``graph``
               False) or as one captured CUDA graph (``graph`` True, what a latency-bound server does)
* ``conv2d``   one int8 convolution, called as an operator with packed weights
* ``conv3d``   one three-dimensional int8 convolution
* ``dense``    one u8 x s8 matrix product
* ``conv_f16`` one fp16 convolution with fp32 results
* ``gemm_f16`` one fp16 matrix product with fp32 results
* ``layout``   NCHW to channel blocks and back, the ends of every blocked chain
"""
from __future__ import annotations

import math

import torch

import unit_b200 as U
from unit_b200 import resnet50 as R


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def _conv2d(name, n, c_in, h, w, c_out, kh, kw, stride, pad_h, pad_w, epilogue, signed, shift, named_out):
    return {'name': name, 'kind': 'conv2d', 'n': n, 'c_in': c_in, 'h': h, 'w': w, 'c_out': c_out, 'kh': kh, 'kw': kw,
            'stride': stride, 'pad_h': pad_h, 'pad_w': pad_w, 'epilogue': epilogue, 'signed': signed, 'shift': shift,
            'named_out': named_out}


def listed():
    return [
        # One image through the network with as little delay as possible: a serving program's smallest batch,
        # replayed as a captured graph.  54 launches in one dependent chain.
        {'name': 'network_b1_graph', 'kind': 'network', 'n': 1, 'graph': True, 'shift': 8},
        # A server's ordinary batch, the plans run one by one.
        {'name': 'network_b32', 'kind': 'network', 'n': 32, 'graph': False, 'shift': 10},
        # Offline inference: the batch the headline figure is quoted on.
        {'name': 'network_b256', 'kind': 'network', 'n': 256, 'graph': False, 'shift': 8},
        # A single small convolution called as an operator (result allocated by the call): 3x3 64->64 at 56x56,
        # s32 result.  Latency: the launch and the host's work around it.
        _conv2d('conv2d_3x3_64_b1', 1, 64, 56, 56, 64, 3, 3, 1, 1, 1, 'raw', False, 8, False),
        # The graph flow's fused operator, (conv + bias) * 11 on signed activations, on a separable 1x7 layer
        # of the shape corpus (17x17, 192 channels: odd sizes everywhere) at a small batch.
        _conv2d('conv2d_1x7_192_b8_signed', 8, 192, 17, 17, 192, 1, 7, 1, 0, 3, 'mul', True, 8, False),
        # The int8 matrix product of a transformer's feed-forward layer on 128 tokens.
        {'name': 'dense_128x3072x768', 'kind': 'dense', 'm': 128, 'n': 3072, 'k': 768},
        # The large int8 matrix product.
        {'name': 'dense_4096', 'kind': 'dense', 'm': 4096, 'n': 4096, 'k': 4096},
        # One image, a strided fp16 layer (128 channels, 56x56 to 28x28).
        {'name': 'conv_f16_3x3s2_128_b1', 'kind': 'conv_f16', 'n': 1, 'c_in': 128, 'h': 56, 'w': 56, 'c_out': 128,
         'k': 3, 'stride': 2, 'pad': 1},
        # The fp16 path's large convolution: 3x3 256->256 at 14x14, batch 256.
        {'name': 'conv_f16_3x3_256_b256', 'kind': 'conv_f16', 'n': 256, 'c_in': 256, 'h': 14, 'w': 14, 'c_out': 256,
         'k': 3, 'stride': 1, 'pad': 1},
        # An fp16 matrix product whose sizes are no multiples of a tile.
        {'name': 'gemm_f16_2500x2064x3080', 'kind': 'gemm_f16', 'm': 2500, 'n': 2064, 'k': 3080},
        # A video batch: 3x3x3 64->64 on 16 frames of 58x58 (already padded).
        {'name': 'conv3d_3x3x3_64_b4', 'kind': 'conv3d', 'n': 4, 'c_in': 64, 'd': 16, 'h': 58, 'w': 58, 'c_out': 64,
         'k': 3, 'stride': 1, 'pad': 0, 'requant': False},
        # fp16 activations from NCHW into channel blocks and back, at an odd image size.
        {'name': 'layout_f16_64x256x35', 'kind': 'layout', 'n': 64, 'c': 256, 'h': 35, 'w': 35, 'c_block': 16,
         'dtype': 'float16'},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_conv2d(rng):
    c_in = 16 * _log_int(rng, 1, 64)
    c_out = 16 * _log_int(rng, 1, 64)
    hw = rng.choice([7, 8, 14, 17, 28, 35, 56, _log_int(rng, 5, 80)])
    kh, kw = rng.choice([(1, 1), (1, 1), (1, 1), (3, 3), (3, 3), (3, 3), (5, 5), (1, 7), (7, 1)])
    stride = rng.choice([1, 1, 1, 2]) if kh == kw else 1
    epilogue = rng.choice(['requant', 'requant', 'raw', 'mul', 'residual'])
    return _conv2d('', _log_int(rng, 1, 128), c_in, hw, hw if rng.random() < 0.8 else hw + rng.randint(1, 6), c_out, kh, kw,
                   stride, kh // 2, kw // 2, epilogue, rng.random() < 0.25, rng.randint(7, 12), rng.random() < 0.5)


def _draw_conv3d(rng):
    k, stride = rng.choice([(3, 1), (3, 1), (3, 2), (1, 2)])
    hw = rng.choice([9, 14, 16, 28, 30, 56, 58])
    return {'kind': 'conv3d', 'n': _log_int(rng, 1, 8), 'c_in': 32 * _log_int(rng, 1, 16), 'd': rng.choice([8, 16, 16, 17]), 'h': hw,
            'w': hw, 'c_out': 32 * _log_int(rng, 1, 16), 'k': k, 'stride': stride, 'pad': rng.choice([0, 0, k // 2]),
            'requant': rng.random() < 0.5}


def _draw_conv_f16(rng):
    k = rng.choice([1, 1, 3, 3, 3, 5])
    return {'kind': 'conv_f16', 'n': _log_int(rng, 1, 256), 'c_in': 16 * _log_int(rng, 2, 64),
            'h': (hw := rng.choice([7, 8, 14, 17, 28, 35, 56])), 'w': hw, 'c_out': 16 * _log_int(rng, 2, 64), 'k': k,
            'stride': rng.choice([1, 1, 1, 2]), 'pad': k // 2}


def _draw_product(rng, kind):
    step = 16 if kind == 'dense' else 8
    return {'kind': kind, 'm': _log_int(rng, 16, 6000), 'n': 16 * _log_int(rng, 4, 320), 'k': step * _log_int(rng, 64 // step, 5120 // step)}


def _draw_layout(rng):
    image = rng.random() < 0.4   # images entering a blocked network (3 channels), or activations inside one
    hw = rng.choice([224, 224, 299, 160]) if image else rng.choice([7, 14, 17, 28, 35, 56])
    return {'kind': 'layout', 'n': _log_int(rng, 1, 128), 'c': 3 if image else _log_int(rng, 16, 1024), 'h': hw, 'w': hw,
            'c_block': 4 if image else 16, 'dtype': rng.choice(['uint8', 'float16', 'int32'])}


def draw(rng):
    """A case of the ranges above, none more expensive than the largest listed one."""
    while True:
        kind = rng.choice(['network', 'conv2d', 'conv2d', 'conv2d', 'dense', 'dense', 'conv_f16', 'conv_f16', 'gemm_f16', 'gemm_f16',
                           'conv3d', 'layout'])
        if kind == 'network':
            case = {'kind': kind, 'n': _log_int(rng, 1, 250), 'graph': rng.random() < 0.5, 'shift': rng.randint(8, 11)}
        elif kind == 'conv2d':
            case = _draw_conv2d(rng)
            del case['name']
        elif kind == 'conv3d':
            case = _draw_conv3d(rng)
        elif kind == 'conv_f16':
            case = _draw_conv_f16(rng)
        elif kind == 'layout':
            case = _draw_layout(rng)
        else:
            case = _draw_product(rng, kind)
        if kind == 'network':
            return case
        w = work(case)
        if w['flops'] <= 4e11 and w['bytes'] <= 6e8:
            return case


# --------------------------------------------------------------------------
# inputs: made on the GPU from the seed, with the distributions of unit_b200.resnet50
# --------------------------------------------------------------------------
class _Source:
    def __init__(self, seed):
        self.gen = torch.Generator(device='cuda').manual_seed(int(seed))

    def activations(self, shape, signed=False):
        """Post-ReLU u8 (half zeros, the rest uniform in [1, 255]); signed ones uniform in [-128, 127]."""
        if signed:
            return torch.randint(-128, 128, shape, dtype=torch.int8, device='cuda', generator=self.gen)
        x = torch.randint(-255, 256, shape, dtype=torch.int16, device='cuda', generator=self.gen)
        return x.clamp_(min=0).to(torch.uint8)

    def weights(self, shape):
        w = torch.randn(shape, device='cuda', generator=self.gen)
        return (w * 32).round_().clamp_(-128, 127).to(torch.int8)

    def bias(self, n):
        return torch.randint(-2 ** 15, 2 ** 15, (n,), dtype=torch.int32, device='cuda', generator=self.gen)

    def matrix(self, shape, lo, hi, dtype):
        return torch.randint(lo, hi, shape, dtype=dtype, device='cuda', generator=self.gen)

    def normal(self, shape, scale=1.0):
        return (torch.randn(shape, device='cuda', generator=self.gen) * scale).to(torch.float16)


def _network_layers():
    """The 53 convolutions in order: (layer, what it reads, whether it ends a block).  Reads: 'image' (the
    stem), 'block' (the block's input) or 'last' (the previous convolution's output)."""
    by_name = {l.name: l for l in R.LAYERS}
    seq = [(by_name['stem_7x7s2_3_64'], 'image', False)]
    stages = [('s1', 3, 's1_1x1_64_64', 's1_3x3_64_64', 's1_proj_64_256', 's1_1x1_256_64', 's1_3x3_64_64', 's1_1x1_64_256'),
              ('s2', 4, 's2_1x1_256_128', 's2_3x3s2_128_128', 's2_proj_s2_256_512', 's2_1x1_512_128', 's2_3x3_128_128',
               's2_1x1_128_512'),
              ('s3', 6, 's3_1x1_512_256', 's3_3x3s2_256_256', 's3_proj_s2_512_1024', 's3_1x1_1024_256', 's3_3x3_256_256',
               's3_1x1_256_1024'),
              ('s4', 3, 's4_1x1_1024_512', 's4_3x3s2_512_512', 's4_proj_s2_1024_2048', 's4_1x1_2048_512', 's4_3x3_512_512',
               's4_1x1_512_2048')]
    for _, blocks, first_reduce, first_3x3, projection, reduce, conv3x3, expand in stages:
        for b in range(blocks):
            if b == 0:
                seq.append((by_name[projection], 'shortcut', False))
            seq.append((by_name[first_reduce if b == 0 else reduce], 'block', False))
            seq.append((by_name[first_3x3 if b == 0 else conv3x3], 'last', False))
            seq.append((by_name[expand], 'last', True))
    return seq


def _prepare_network(case, src):
    n, shift = case['n'], case['shift']
    image = src.activations((n, 1, 224, 224, 4))
    image[..., 3] = 0
    # (the stem's output would pass a pooling layer, which is no part of this library: the blocks start from
    # 64 channels at 56x56 of their own)
    block = src.activations((n, 4, 56, 56, 16))
    plans, outputs, keep = [], [], []
    last = shortcut = None
    for layer, reads, ends in _network_layers():
        x = {'image': image, 'block': block, 'shortcut': block, 'last': last}[reads]
        w = src.weights((layer.c_out // 16, layer.c_in_stored // layer.c_block, layer.k, layer.k, layer.c_block // 4, 16, 4))
        packed = U.pack_conv_weights_int8(w, layer.stride, layer.pad)
        bias = src.bias(layer.c_out)
        residual = None
        if ends:
            residual = shortcut if shortcut is not None else block
        plan = U.conv2d_NCHWc_int8_plan(x, packed, stride=layer.stride, padding=layer.pad, bias=bias, out_dtype='uint8',
                                        requant_shift=shift, residual=residual)
        plans.append(plan)
        keep.append(packed)
        if reads == 'image':
            outputs.append(plan.out)
        elif reads == 'shortcut':
            shortcut = plan.out
        else:
            last = plan.out
        if ends:
            block, shortcut = plan.out, None
    outputs.append(block)
    state = {'kind': 'network', 'plans': plans, 'outputs': outputs, 'keep': keep, 'graph': None}
    if case['graph']:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for p in plans:   # once before the capture: first launches look kernels up
                p.run()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for p in plans:
                p.run()
        state['graph'] = graph
    return state


def _out_size(size, k, stride, pad):
    return (size + 2 * pad - k) // stride + 1


def prepare(case, seed):
    """Inputs, packed weights and plans: what a program holds before the call."""
    src = _Source(seed)
    kind = case['kind']
    if kind == 'network':
        return _prepare_network(case, src)
    state = {'kind': kind}
    if kind == 'conv2d':
        n, ci, co = case['n'], case['c_in'], case['c_out']
        stride, pad = case['stride'], (case['pad_h'], case['pad_w'])
        state['x'] = src.activations((n, ci // 16, case['h'], case['w'], 16), case['signed'])
        w = src.weights((co // 16, ci // 16, case['kh'], case['kw'], 4, 16, 4))
        state['w'] = U.pack_conv_weights_int8(w, stride, pad)
        oshape = (n, co // 16, _out_size(case['h'], case['kh'], stride, pad[0]), _out_size(case['w'], case['kw'], stride, pad[1]), 16)
        options = {'stride': stride, 'padding': pad}
        if case['epilogue'] != 'raw':
            options['bias'] = src.bias(co)
        if case['epilogue'] == 'mul':
            options['mul'] = 11
        if case['epilogue'] in ('requant', 'residual'):
            options.update(out_dtype='uint8', requant_shift=case['shift'])
        if case['epilogue'] == 'residual':
            options['residual'] = src.activations(oshape)
        if case['named_out']:
            options['out'] = torch.empty(oshape, dtype=torch.uint8 if case['epilogue'] in ('requant', 'residual') else torch.int32,
                                         device='cuda')
        state['options'] = options
    elif kind == 'conv3d':
        n, ci, co, k = case['n'], case['c_in'], case['c_out'], case['k']
        state['x'] = src.activations((n, ci // 16, case['d'], case['h'], case['w'], 16))
        state['w'] = U.pack_conv3d_weights_int8(src.weights((co // 16, ci // 16, k, k, k, 4, 16, 4)), case['stride'])
        state['options'] = {'stride': case['stride'], 'padding': case['pad']}
        if case['requant']:
            state['options'].update(bias=src.bias(co), requant_shift=10)
    elif kind == 'dense':
        m, n, k = case['m'], case['n'], case['k']
        state['x'] = src.matrix((m, k), 0, 256, torch.uint8)
        state['w'] = U.pack_dense_weights_int8(src.matrix((n // 16, k // 4, 16, 4), -128, 128, torch.int8))
    elif kind == 'gemm_f16':
        state['x'] = src.normal((case['m'], case['k']))
        state['w'] = U.pack_gemm_weights_f16(src.normal((case['k'], case['n']), 0.05))
    elif kind == 'conv_f16':
        k = case['k']
        state['x'] = src.normal((case['n'], case['c_in'] // 16, case['h'], case['w'], 16))
        state['w'] = U.pack_conv_weights_f16(src.normal((case['c_out'] // 16, case['c_in'] // 16, k, k, 16, 16), 0.05))
        state['stride'], state['pad'] = case['stride'], case['pad']
    else:
        shape = (case['n'], case['c'], case['h'], case['w'])
        if case['dtype'] == 'float16':
            state['x'] = src.normal(shape)
        elif case['dtype'] == 'uint8':
            state['x'] = src.activations(shape)
        else:
            state['x'] = src.matrix(shape, -2 ** 30, 2 ** 30, torch.int32)
        state['c'], state['c_block'] = case['c'], case['c_block']
    return state


def run(state):
    """One pass through the public operators."""
    kind = state['kind']
    if kind == 'network':
        if state['graph'] is not None:
            state['graph'].replay()
        else:
            for plan in state['plans']:
                plan.run()
        return state['outputs']
    if kind == 'conv2d':
        return U.conv2d_NCHWc_int8(state['x'], state['w'], **state['options'])
    if kind == 'conv3d':
        return U.conv3d_NCDHWc_int8(state['x'], state['w'], **state['options'])
    if kind == 'dense':
        return U.dense_dotprod(state['x'], state['w'])
    if kind == 'gemm_f16':
        return U.gemm_f16f32(state['x'], state['w'])
    if kind == 'conv_f16':
        return U.conv2d_NCHW16c_OHWI16o(state['x'], state['w'], state['stride'], state['stride'], padding=state['pad'])
    blocked = U.pack_data_nchwc(state['x'], state['c_block'])
    return blocked, U.unpack_data_nchwc(blocked, state['c'])


# --------------------------------------------------------------------------
# what a pass cannot do without, and how close two results have to be
# --------------------------------------------------------------------------
def work(case):
    """Bytes (every input read once, every output written once) and operations (two per multiply-accumulate)."""
    kind = case['kind']
    if kind == 'network':
        n, total, ops = case['n'], 0.0, 0.0
        for layer, _, ends in _network_layers():
            total += layer.bytes(n) + (n * layer.c_out * layer.out_hw ** 2 if ends else 0)
            ops += layer.ops(n)
        return {'bytes': total, 'flops': ops}
    if kind == 'conv2d':
        oh = _out_size(case['h'], case['kh'], case['stride'], case['pad_h'])
        ow = _out_size(case['w'], case['kw'], case['stride'], case['pad_w'])
        out = case['n'] * oh * ow * case['c_out']
        taps = case['kh'] * case['kw']
        x = case['n'] * case['c_in'] * case['h'] * case['w']
        per_out = {'raw': 4, 'mul': 4, 'requant': 1, 'residual': 2}[case['epilogue']]
        return {'bytes': float(x + case['c_in'] * case['c_out'] * taps + out * per_out + 4 * case['c_out']),
                'flops': 2.0 * out * case['c_in'] * taps}
    if kind == 'conv3d':
        k, s, p = case['k'], case['stride'], case['pad']
        out = case['n'] * case['c_out'] * _out_size(case['d'], k, s, p) * _out_size(case['h'], k, s, p) * _out_size(case['w'], k, s, p)
        x = case['n'] * case['c_in'] * case['d'] * case['h'] * case['w']
        return {'bytes': float(x + case['c_in'] * case['c_out'] * k ** 3 + out * (1 if case['requant'] else 4)),
                'flops': 2.0 * out * case['c_in'] * k ** 3}
    if kind in ('dense', 'gemm_f16'):
        m, n, k, eb = case['m'], case['n'], case['k'], 1 if kind == 'dense' else 2
        return {'bytes': float((m * k + n * k) * eb + 4 * m * n), 'flops': 2.0 * m * n * k}
    if kind == 'conv_f16':
        k, s, p = case['k'], case['stride'], case['pad']
        out = case['n'] * case['c_out'] * _out_size(case['h'], k, s, p) * _out_size(case['w'], k, s, p)
        x = case['n'] * case['c_in'] * case['h'] * case['w']
        return {'bytes': 2.0 * (x + case['c_in'] * case['c_out'] * k * k) + 4.0 * out, 'flops': 2.0 * out * case['c_in'] * k * k}
    eb = {'uint8': 1, 'float16': 2, 'int32': 4}[case['dtype']]
    cb = case['c_block']
    plane = case['n'] * case['h'] * case['w']
    blocked = (case['c'] + cb - 1) // cb * cb
    # pack reads c and writes the padded blocks, unpack reads the blocks that hold channels and writes c
    return {'bytes': 2.0 * plane * (case['c'] + blocked) * eb, 'flops': 0.0}


def tolerance(case):
    """Integers and moved bytes are exact; fp16 products summed in fp32 depend on the order of the sum."""
    if case['kind'] in ('gemm_f16', 'conv_f16'):
        return {'rel': 2e-5}
    return 'exact'
