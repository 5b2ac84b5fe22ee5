"""What a program that uses this framework has it do, as cases that can be timed and compared.

One GPU, one rank (`group=None`): the expert-parallel layer on the experts of that rank, the router frontend, and the
load-time weight transform, each through the package's public functions. `listed()` are the standing cases, `draw(rng)`
gives more of the same ranges.

A case is a dict of plain values:

  path      'layer'     routed, quantised tokens lie in the buffer's views; one `fp4_fp4_mega_moe` / `fp8_fp4_mega_moe`
            'hidden'    bf16 hidden states; router, top-8, quantisation and the layer in one `mega_moe_from_hidden`
            'frontend'  bf16 hidden states; router, top-8 and quantisation alone (`fe_forward` into the buffer's views)
            'load'      packed expert weights and their scale words; one `transform_weights_for_mega_moe`
  fmt       'mxfp4', 'nvfp4' (with per-tensor global scales) or 'fp8' (E4M3 tokens, MXFP4 weights)
  tokens    tokens of the call; `capacity` is what the buffer was created for (a server's largest batch)
  experts, hidden, inter, topk    the layer's geometry
  masked    share of routing slots that are switched off (-1), as padding and dropped tokens are
  clamp     SwiGLU clamp, negative for none
  scores    'softmax', or 'sigmoid' with a Zipf(1.2) expert bias: a few hot experts receive many rows
"""
import math

import torch

import hopper_megamoe_basedondeepgemm_b200 as mm
from hopper_megamoe_basedondeepgemm_b200 import quant
from hopper_megamoe_basedondeepgemm_b200 import workload as W

# the benchmark's layer: 48 experts on the rank, H = 3072, I = 1280, top-8
LAYER = dict(experts=48, hidden=3072, inter=1280, topk=8)
# the small layer of the smoke run and the tests
SMALL = dict(experts=8, hidden=1024, inter=512, topk=4)
LARGEST_EXPERT, LARGEST_LAYER = 3072 * 1280, 48 * 3072 * 1280      # no drawn layer is larger than the benchmark's
MAX_ROWS = 4096                                 # routed rows one launch takes


def _case(name, path, fmt, tokens, capacity, geometry, masked=0.0, clamp=10.0, scores='softmax'):
    c = dict(path=path, fmt=fmt, tokens=tokens, capacity=capacity, masked=masked, clamp=clamp, scores=scores, **geometry)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a layer small enough for its launch latency to be all there is
        _case('small layer, 6 tokens', 'layer', 'mxfp4', 6, 16, SMALL),
        # decode: one request, the smallest step a server takes
        _case('decode 1, mxfp4', 'layer', 'mxfp4', 1, 16, LAYER),
        # decode with E4M3 activations, two requests
        _case('decode 2, fp8', 'layer', 'fp8', 2, 16, LAYER),
        # decode of an odd batch, NVFP4 with global scales
        _case('decode 13, nvfp4', 'layer', 'nvfp4', 13, 16, LAYER),
        # an ordinary batch
        _case('batch 64, mxfp4', 'layer', 'mxfp4', 64, 64, LAYER),
        # a ragged batch with E4M3 activations and padding slots
        _case('batch 100, fp8', 'layer', 'fp8', 100, 128, LAYER, masked=0.1),
        # a prefill chunk that does not fill the buffer, no clamp
        _case('prefill 300, nvfp4', 'layer', 'nvfp4', 300, 512, LAYER, clamp=-1.0),
        # the largest launch: 4096 routed rows
        _case('prefill 512, mxfp4', 'layer', 'mxfp4', 512, 512, LAYER),
        # decode from hidden states in a single launch
        _case('hidden 1, mxfp4', 'hidden', 'mxfp4', 1, 16, LAYER),
        # a skewed batch from hidden states: sigmoid scores and a biased router
        _case('hidden 96, nvfp4, skewed', 'hidden', 'nvfp4', 96, 128, LAYER, scores='sigmoid'),
        # the router frontend as a call of its own, at the width of eight ranks' experts
        _case('frontend 8 of 384', 'frontend', 'mxfp4', 8, 64, dict(LAYER, experts=384)),
        # what a server does once per layer when it loads a model
        _case('load, mxfp4', 'load', 'mxfp4', 0, 0, LAYER),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(['layer', 'layer', 'layer', 'layer', 'layer', 'hidden', 'hidden', 'frontend', 'load'])
    fmt = rng.choice(['mxfp4', 'mxfp4', 'nvfp4', 'fp8'])
    if path == 'frontend':
        geometry = dict(experts=rng.choice([16, 48, 64, 128, 192, 256, 384]), hidden=512 * rng.randint(2, 8), inter=1280, topk=8)
        tokens = _log_int(rng, 1, 64)
        return _case(None, path, fmt, tokens, 64, geometry)
    if path == 'load':
        geometry = dict(experts=rng.randint(8, 48), hidden=512 * rng.randint(2, 6), inter=256 * rng.randint(1, 5), topk=8)
        return _case(None, path, rng.choice(['mxfp4', 'nvfp4']), 0, 0, geometry)
    geometry = dict(LAYER)
    if rng.random() < 0.5:
        while True:
            geometry = dict(experts=rng.choice([8, 12, 16, 24, 32, 48, 64]), hidden=512 * rng.randint(2, 8),
                            inter=256 * rng.randint(1, 8), topk=8 if path == 'hidden' else rng.choice([2, 4, 6, 8]))
            size = geometry['hidden'] * geometry['inter']
            if size <= LARGEST_EXPERT and geometry['experts'] * size <= LARGEST_LAYER:
                break
    tokens = _log_int(rng, 1, (256 if path == 'hidden' else MAX_ROWS // 8))
    capacity = max(16, 1 << (tokens - 1).bit_length())
    return _case(None, path, fmt, tokens, capacity, geometry,
                 masked=rng.choice([0.0, 0.0, 0.1]) if path == 'layer' else 0.0, clamp=rng.choice([-1.0, 10.0, round(rng.uniform(4.0, 20.0), 2)]),
                 scores=rng.choice(['softmax', 'sigmoid']) if path == 'hidden' else 'softmax')


def _routing(case, seed):
    """Distinct experts per token, uniform; softmax weights; some slots switched off."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    scores = torch.randn((case['tokens'], case['experts']), generator=g, device='cuda')
    w, idx = torch.topk(scores, case['topk'], dim=-1)
    w = torch.softmax(w, dim=-1)
    off = torch.rand(idx.shape, generator=g, device='cuda') < case['masked']
    return idx.masked_fill(off, -1), w.masked_fill(off, 0.0).float()


def _packed_weights(case, seed):
    """bf16 expert weights ~ N(0, 0.02) as a checkpoint holds them: packed E2M1 and MN-major scale words, and the
    per-tensor global scales (1 unless NVFP4)."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    out, scales = [], []
    for n, k in ((2 * case['inter'], case['hidden']), (case['hidden'], case['inter'])):
        w = (torch.randn((case['experts'], n, k), generator=g, device='cuda') * 0.02).to(torch.bfloat16)
        gs = mm.nvfp4_global_scale(w) if case['fmt'] == 'nvfp4' else 1.0
        out.append(quant.cast_grouped_weights_to_fp4(w, case['fmt'], gs))
        scales.append(gs)
    return out, scales


def prepare(case, seed):
    c, s = case, dict(case=case)
    t, h, e = c['tokens'], c['hidden'], c['experts']
    if c['path'] in ('layer', 'hidden', 'load'):
        (w1, w2), (s['gs1'], s['gs2']) = _packed_weights(c, seed)
        if c['path'] == 'load':
            s['w1'], s['w2'] = w1, w2
            return s
        s['l1'], s['l2'] = mm.transform_weights_for_mega_moe(w1, w2)
        s['buf'] = mm.get_symm_buffer_for_mega_moe(None, e, c['capacity'], c['topk'], h, c['inter'], act_format=c['fmt'])
        s['y'] = torch.empty((t, h), dtype=torch.bfloat16, device='cuda')
        s['stats'] = torch.zeros(e, dtype=torch.int32, device='cuda')
    s['x_gs'], s['mid_gs'] = (1.0 / 64.0, 1.0 / 512.0) if c['fmt'] == 'nvfp4' else (1.0, 1.0)
    if c['path'] == 'layer':
        _, xq, xsf = W.make_tokens(t, h, c['fmt'], seed + 1, global_scale=s['x_gs'])
        idx, tw = _routing(c, seed + 2)
        b = s['buf']
        b.x[:t].copy_(xq); b.x_sf[:t].copy_(xsf); b.topk_idx[:t].copy_(idx); b.topk_weights[:t].copy_(tw)
        return s
    g = torch.Generator(device='cuda').manual_seed(seed + 1)
    s['hidden'] = torch.randn((t, h), generator=g, device='cuda').to(torch.bfloat16)
    s['router'] = (torch.randn((e, h), generator=g, device='cuda') / h ** 0.5).to(torch.bfloat16)
    if c['path'] == 'frontend':
        # the views of a buffer, as plain tensors: the frontend needs nothing else of it
        vec = quant.SF_VEC[c['fmt']]
        s['x'] = torch.zeros((t, h if c['fmt'] == 'fp8' else h // 2), dtype=torch.float8_e4m3fn if c['fmt'] == 'fp8' else torch.int8, device='cuda')
        s['x_sf'] = torch.zeros((t, h // (4 * vec)), dtype=torch.int32, device='cuda')
        s['idx'] = torch.zeros((t, c['topk']), dtype=torch.int64, device='cuda')
        s['tw'] = torch.zeros((t, c['topk']), dtype=torch.float32, device='cuda')
        s['ws'] = torch.zeros(mm.fe_workspace_bytes(e), dtype=torch.uint8, device='cuda')
        s['mode'] = {'fp8': 2, 'mxfp4': 3, 'nvfp4': 4}[c['fmt']]
        return s
    s['ws'] = torch.zeros(mm.fe_workspace_bytes(s['buf']), dtype=torch.uint8, device='cuda')
    s['bias'] = None
    if c['scores'] == 'sigmoid':
        order = torch.randperm(e, generator=g, device='cuda')
        s['bias'] = (1.0 / torch.arange(1, e + 1, dtype=torch.float32, device='cuda') ** 1.2)[order].contiguous()
    return s


def run(s):
    c = s['case']
    clamp = c['clamp'] if c['clamp'] >= 0 else None
    if c['path'] == 'load':
        (a, _), (b, _) = mm.transform_weights_for_mega_moe(s['w1'], s['w2'])
        return a, b
    if c['path'] == 'frontend':
        mm.fe_forward(s['hidden'], s['router'], s['x'], s['x_sf'], s['idx'], s['tw'], s['ws'], s['mode'])
        return s['x'].view(torch.int8), s['x_sf'], s['idx'], s['tw']
    if c['path'] == 'hidden':
        mm.mega_moe_from_hidden(s['y'], s['hidden'], s['router'], s['l1'], s['l2'], s['buf'], s['ws'],
                                cumulative_local_expert_recv_stats=s['stats'], activation_clamp=clamp,
                                score_mode=0 if s['bias'] is None else 1, expert_bias=s['bias'], x_global_scale=s['x_gs'],
                                l1_global_scale=s['gs1'], l2_global_scale=s['gs2'], mid_global_scale=s['mid_gs'])
        t = c['tokens']
        return s['y'], s['stats'], s['buf'].topk_idx[:t], s['buf'].topk_weights[:t]
    if c['fmt'] == 'fp8':
        mm.fp8_fp4_mega_moe(s['y'], s['l1'], s['l2'], s['buf'], cumulative_local_expert_recv_stats=s['stats'], activation_clamp=clamp)
    else:
        mm.fp4_fp4_mega_moe(s['y'], s['l1'], s['l2'], s['buf'], cumulative_local_expert_recv_stats=s['stats'], activation_clamp=clamp,
                            x_global_scale=s['x_gs'], l1_global_scale=s['gs1'], l2_global_scale=s['gs2'], mid_global_scale=s['mid_gs'])
    return s['y'], s['stats']


def work(case):
    c = case
    t, h, i, e, k = c['tokens'], c['hidden'], c['inter'], c['experts'], c['topk']
    per_expert = W.weight_bytes_per_expert(h, i, c['fmt'])
    if c['path'] == 'load':
        return {'bytes': 2 * e * per_expert, 'flops': 0}
    vec = quant.SF_VEC[c['fmt']]
    row = (h if c['fmt'] == 'fp8' else h // 2) + h // vec           # one quantised token and its scale bytes
    routing = t * k * 12                                            # int64 expert and float weight per slot
    if c['path'] == 'frontend':
        return {'bytes': e * h * 2 + t * (h * 2 + row) + routing, 'flops': 2 * t * e * h}
    # experts with at least one row: expected number under uniform routing (an upper bound for the skewed one)
    live = e * (1.0 - (1.0 - k / e * (1.0 - c['masked'])) ** t)
    out = {'bytes': live * per_expert + routing + t * h * 2, 'flops': 2 * t * k * (1.0 - c['masked']) * 3 * h * i}
    out['bytes'] += e * h * 2 + t * (h * 2 + row) if c['path'] == 'hidden' else t * row
    out['flops'] += 2 * t * e * h if c['path'] == 'hidden' else 0
    return out


def tolerance(case):
    if case['path'] == 'load':
        return 'exact'
    if case['path'] == 'frontend':
        return {'rel': 1e-5, 'max': 1e-4, 'differ': 0.0}            # fp32 routing weights; bytes and expert ids are exact
    # bf16 outputs; a sum in another order can move single E2M1 / E4M3 codes of the intermediate
    return {'rel': 1e-2, 'max': 0.2, 'differ': 0.0}
