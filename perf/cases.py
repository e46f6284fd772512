"""Cases for timing this package as its users call it: the layer's forward from one row (a decode step) to a few
thousand (a prompt or an evaluation batch), the forward on host buffers, the dense weight, and a decode step of decoder
blocks.  Every input comes from a seed: Bernoulli(0.5) bits, N(0, 0.02) coefficients, N(0, 1) activations.

A case is a dict.  kind "forward", "host" and "weight" describe one layer: out = rw*P and in = cw*Q features, `bits` bit
layers, patches P x Q of rank r, m rows of X, element type, bias or not.  kind "block" is `layers` decoder blocks at
one new token for each of `batch` sequences with `context` tokens in the cache."""
import math

import torch

from bqq_b200 import BinaryQuadratic
from bqq_b200.decoder_stack import DecoderLayer, StackConfig

DTYPES = {'f32': torch.float32, 'bf16': torch.bfloat16, 'f16': torch.float16}
MAX_FLOPS = 7.0e10           # a drawn case costs no more than the largest listed one
MAX_BIT_ENTRIES = 3 * 8192 * 28672


def _layer(kind, rw, cw, bits, P=32, Q=32, r=32, m=1, dtype='bf16', bias=False, name=None):
    case = dict(kind=kind, rw=rw, cw=cw, bits=bits, P=P, Q=Q, r=r, m=m, dtype=dtype, bias=bias)
    return case if name is None else dict(case, name=name)


def _block(layers, hidden, intermediate, heads, kv_heads, bits, batch, context, name=None):
    case = dict(kind='block', layers=layers, hidden=hidden, intermediate=intermediate, heads=heads, kv_heads=kv_heads,
                bits=bits, batch=batch, context=context)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # one token through a small attention projection: latency and launches
        _layer('forward', 64, 64, 2, name='decode_2048x2048_b2_m1'),
        # one token through the widest MLP projection of the decode sweep: streaming the planes
        _layer('forward', 128, 448, 4, name='decode_4096x14336_b4_m1'),
        # a few sequences decoded together, 4 and 16 rows
        _layer('forward', 192, 64, 3, m=4, name='decode_6144x2048_b3_m4'),
        _layer('forward', 128, 448, 3, m=16, name='decode_4096x14336_b3_m16'),
        # patches that fill no block of 32, an odd number of col patches, a bias, fp16 activations
        _layer('forward', 21, 51, 3, P=96, Q=40, r=33, m=5, dtype='f16', bias=True, name='decode_ragged_2016x2040_b3_m5'),
        # a serving batch on the large bit-depth-extended layer (2 + 1 bit layers, rank 64)
        _layer('forward', 128, 448, 3, P=64, Q=64, r=64, m=32, name='batch_8192x28672_b3_r64_m32'),
        # a serving batch of 64 sequences through an output projection
        _layer('forward', 128, 128, 2, m=64, name='batch_4096x4096_b2_m64'),
        # a prompt of 2048 tokens
        _layer('forward', 128, 128, 2, m=2048, name='prefill_4096x4096_b2_m2048'),
        # an evaluation batch in fp32, rows not a multiple of any tile, with a bias
        _layer('forward', 64, 64, 3, m=333, dtype='f32', bias=True, name='eval_2048x2048_b3_m333_f32'),
        # a serving loop that keeps its activations in pinned host buffers
        _layer('host', 64, 192, 3, name='host_2048x6144_b3_m1'),
        # one decode step of two blocks of the 8B decoder stack after a 512-token prompt, replayed from a graph
        _block(2, 4096, 14336, 32, 8, 2, 1, 512, name='block_step_8b_m1'),
        # dequantising a layer (the builder's route back to a dense model)
        _layer('weight', 128, 448, 4, name='weight_4096x14336_b4_bf16'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['forward'] * 7 + ['host', 'weight', 'block'])
    if kind == 'block':
        kv = rng.choice([1, 2, 4, 8])
        heads = min(32, kv * rng.choice([1, 2, 4, 8]))
        hidden = heads * 128
        inter = 32 * _log_int(rng, hidden // 32, 3.5 * hidden // 32)
        return _block(rng.choice([1, 2]), hidden, inter, heads, kv, rng.choice([2, 2, 3, 4]), _log_int(rng, 1, 64),
                      _log_int(rng, 16, 1000))
    while True:
        P, Q, r = rng.choice([(32, 32, 32)] * 6 + [(64, 64, 64), (64, 64, 32), (64, 64, 32)] + [None] * 2) or (
            rng.choice([16, 24, 40, 96, 128]), rng.choice([16, 24, 40, 96, 128]), rng.choice([7, 12, 16, 33, 64]))
        rw = max(1, round(_log_int(rng, 256, 28672) / P))
        cw = max(1, round(_log_int(rng, 256, 28672) / Q))
        m = {'forward': _log_int(rng, 1, 4096), 'host': _log_int(rng, 1, 64), 'weight': 1}[kind]
        case = _layer(kind, rw, cw, rng.choice([1, 2, 2, 3, 4]), P, Q, r, m,
                      rng.choice(['bf16', 'bf16', 'bf16', 'f16', 'f32']), rng.random() < 0.3)
        if work(case)['flops'] <= MAX_FLOPS and case['bits'] * rw * P * cw * Q <= MAX_BIT_ENTRIES:
            return case


def _make_layer(case, gen):
    grid = (case['bits'], case['rw'], case['cw'])
    bit = lambda *shape: torch.rand(*grid, *shape, generator=gen, device='cuda') < 0.5  # noqa: E731
    A = torch.randn(*grid, 4, generator=gen, device='cuda') * 0.02
    bias = torch.randn(case['rw'] * case['P'], generator=gen, device='cuda') if case['bias'] else None
    layer = BinaryQuadratic(bit(case['P'], case['r']), bit(case['r'], case['Q']), A, bias)
    layer._ensure_packed()                      # bit planes are laid out once per layer, when it is loaded
    return layer


_capture_stream = None


def _make_block(case, gen):
    """Decoder blocks, their caches and one decode step captured as a CUDA graph, as a decode loop keeps them."""
    global _capture_stream
    B, n = case['batch'], case['context']
    cfg = StackConfig(layers=case['layers'], hidden=case['hidden'], intermediate=case['intermediate'], heads=case['heads'],
                      kv_heads=case['kv_heads'], bit_width=case['bits'], max_seq=1024)
    dev = torch.device('cuda', torch.cuda.current_device())
    blocks = [DecoderLayer(cfg, dev, gen, 0, 1) for _ in range(cfg.layers)]
    with torch.no_grad():                       # smaller random weights: projections of normalised rows stay O(1)
        for p in (p for block in blocks for proj in block.children() for p in proj.parameters()):
            p.mul_(0.1)
    cache = torch.zeros(cfg.layers, 2, B, cfg.max_seq, cfg.kv_heads, cfg.head_dim, device=dev, dtype=torch.bfloat16)
    cache[:, :, :, :n].copy_(torch.randn(cfg.layers, 2, B, n, cfg.kv_heads, cfg.head_dim, generator=gen, device=dev))
    x = torch.randn(B, 1, cfg.hidden, generator=gen, device=dev).to(torch.bfloat16)
    inv = 1.0 / (cfg.rope_theta ** (torch.arange(0, cfg.head_dim, 2, device=dev).float() / cfg.head_dim))
    ang = torch.arange(cfg.max_seq, device=dev).float()[:, None] * inv[None, :]
    fa = (ang.cos().to(torch.bfloat16), ang.sin().to(torch.bfloat16), torch.full((B,), n, dtype=torch.int32, device=dev))
    pos = torch.full((1,), n, dtype=torch.int64, device=dev)

    def step():
        h = x
        for i, block in enumerate(blocks):
            h = block(h, cache[i, 0], cache[i, 1], pos, None, None, fa=fa)
        return h

    if _capture_stream is None:
        _capture_stream = torch.cuda.Stream()
    _capture_stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(_capture_stream), torch.no_grad():
        step()                                  # scratch buffers reach their size outside the capture
        _capture_stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=_capture_stream):
            y = step()
    torch.cuda.current_stream().wait_stream(_capture_stream)
    return {'kind': 'block', 'graph': graph, 'y': y, 'cache': cache, 'keep': (blocks, x, fa, pos)}


def prepare(case, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    if case['kind'] == 'block':
        return _make_block(case, gen)
    dtype = DTYPES[case['dtype']]
    layer = _make_layer(case, gen)
    state = {'kind': case['kind'], 'layer': layer, 'dtype': dtype}
    if case['kind'] != 'weight':
        state['x'] = torch.randn(case['m'], case['cw'] * case['Q'], generator=gen, device='cuda').to(dtype)
    if case['kind'] == 'host':
        host = torch.empty(state['x'].shape, dtype=dtype, pin_memory=True)
        host.copy_(state['x'])
        with torch.no_grad():
            state['run'], _ = layer.bind_host(host)
    return state


@torch.no_grad()
def run(state):
    kind = state['kind']
    if kind == 'forward':
        return state['layer'](state['x'])
    if kind == 'host':
        return state['run']()
    if kind == 'weight':
        return state['layer'].get_weight(state['dtype'])
    state['graph'].replay()
    return {'hidden': state['y'], 'cache': state['cache']}


def _layer_work(rw, cw, bits, P, Q, r, m, esize):
    """Bytes: packed bits, fp32 coefficients, x and y.  Operations: the cheaper of the factored form (Z x, then Y u, for
    every bit layer) and the rebuilt dense weight followed by a matrix product."""
    nbytes = bits * rw * cw * r * (P + Q) / 8 + 4 * rw * cw * (3 * bits + 1) + m * (rw * P + cw * Q) * esize
    rebuild = 2.0 * bits * rw * cw * P * Q * r
    dense = 2.0 * m * rw * P * cw * Q
    factored = 2.0 * m * bits * rw * cw * r * (P + Q)
    return nbytes, min(factored, rebuild + dense), rebuild


def work(case):
    if case['kind'] == 'block':
        h, i, hd = case['hidden'], case['intermediate'], 128
        qkv = (case['heads'] + 2 * case['kv_heads']) * hd
        B, n = case['batch'], case['context'] + 1
        parts = [_layer_work(o // 32, k // 32, case['bits'], 32, 32, 32, B, 2) for o, k in
                 ((qkv, h), (h, h), (2 * i, h), (h, i))]
        nbytes = sum(p[0] for p in parts) + B * n * 2 * case['kv_heads'] * hd * 2
        flops = sum(p[1] for p in parts) + 4.0 * B * n * case['heads'] * hd
        return {'bytes': case['layers'] * nbytes, 'flops': case['layers'] * flops}
    esize = 4 if case['dtype'] == 'f32' else 2
    args = [case[k] for k in ('rw', 'cw', 'bits', 'P', 'Q', 'r')]
    if case['kind'] == 'weight':
        nbytes, _, rebuild = _layer_work(*args, 0, esize)
        return {'bytes': nbytes + case['rw'] * case['P'] * case['cw'] * case['Q'] * esize, 'flops': rebuild}
    nbytes, flops, _ = _layer_work(*args, case['m'], esize)
    return {'bytes': nbytes, 'flops': flops}


def tolerance(case):
    if case['kind'] == 'block':
        return {'rel': 1e-2, 'max': 0.2}        # bf16 hidden states rounded after every projection
    if case['dtype'] == 'f32':                  # the forward computes in fewer than 32 bits: 16-bit activations in block
        return {'rel': 1e-5 if case['kind'] == 'weight' else 1e-4, 'max': 1e-3}   # fixed point, or pairs of bf16
    return {'rel': 5e-3 if case['dtype'] == 'bf16' else 1e-3, 'max': 0.03}
