"""The work a user of this package has it do, as cases to time and compare.

A case names a model shape of vesta_gpu_b200.shapes, one of the public calls of VestaGPT2 and its sizes:

  call='step'      a serving loop on device buffers: the scheduled tokens and positions are copied into `x` and `t`, then
                   `step(steps)` runs that many decode steps (the model feeds itself between them)
  call='host'      a loop on host buffers: `steps` calls of `step_host`, every chosen token read on the host and fed back
  call='prefill'   `prefill(tokens, lengths)`: whole prompts into the cache, the first token of every answer

Decode cases start with `ctx` positions in the cache (ragged: from `lo` to `ctx`, one length per sequence); prefill cases
read prompts of `ctx` tokens (ragged: from `lo` to `ctx`). The cache always has room for the whole position table, as a server
would allocate it. Weights have GPT-2's proportions: matrices N(0, 0.02), the two projections into the residual stream smaller
by sqrt(2 L), embeddings wide enough (0.1) that a token is chosen by a clear margin, as in a trained model; so the tokens of two
correct implementations are the same, and logits and cache show how far they are apart.
"""
import math

import numpy as np
import torch

from vesta_gpu_b200.gpt2 import VestaGPT2
from vesta_gpu_b200.shapes import SHAPES

CACHE_STD = 0.5          # K and V of a random-weight layer: LayerNorm output (unit variance) times N(0, 0.02) columns


def _case(name, model, call, batch, ctx, lo=0, steps=1):
    return dict(name=name, model=model, call=call, batch=batch, ctx=ctx, lo=lo or ctx, steps=steps)


def listed():
    return [
        # the smallest call: one interactive user, a short context, one token at a time
        _case('small step b1', 'gpt2', 'step', 1, 37),
        # a loop whose tokens live on the host (sampling, stop words), eight users, an odd context
        _case('small host loop b8', 'gpt2', 'host', 8, 201, steps=4),
        # the ordinary generation of bench.py: eight sequences after 128-token prompts, sixteen tokens per call
        _case('small generate b8', 'gpt2', 'step', 8, 128, steps=16),
        # a partly filled server: an odd number of sequences, each at its own position
        _case('small ragged b23', 'gpt2', 'step', 23, 700, lo=65, steps=4),
        # 64 sequences after 512-token prompts
        _case('small generate b64', 'gpt2', 'step', 64, 512, steps=4),
        # the full batch of one GPU: 256 sequences, ragged contexts of 64 to 512 positions
        _case('small ragged b256', 'gpt2', 'step', 256, 512, lo=64, steps=4),
        # the XL shape, one user and sixteen
        _case('xl step b1', 'gpt2_xl', 'step', 1, 128),
        _case('xl generate b16', 'gpt2_xl', 'step', 16, 128, steps=4),
        # time to the first token: one prompt of an odd length, eight of 128 tokens, 64 ragged ones of up to 512, a few at the XL shape
        _case('small prefill 1x77', 'gpt2', 'prefill', 1, 77),
        _case('small prefill 8x128', 'gpt2', 'prefill', 8, 128),
        _case('small prefill 64 ragged', 'gpt2', 'prefill', 64, 512, lo=64),
        _case('xl prefill 4 ragged', 'gpt2_xl', 'prefill', 4, 250, lo=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = 'gpt2_xl' if rng.random() < 0.25 else 'gpt2'
    call = rng.choices(('step', 'host', 'prefill'), (0.5, 0.15, 0.35))[0]
    limit = max(_weight(work(c)) for c in listed())
    while True:
        ragged = rng.random() < 0.5
        if call == 'prefill':
            batch, ctx, steps = _log(rng, 1, 64), _log(rng, 8, 900), 1
        else:
            batch = _log(rng, 1, (256 if model == 'gpt2' else 32) if call == 'step' else 16)
            ctx, steps = _log(rng, 8, 1000), _log(rng, 1, 16 if model == 'gpt2' else 4)
        lo = max(1, ctx // rng.randint(2, 9)) if ragged and batch > 1 else ctx
        case = dict(model=model, call=call, batch=batch, ctx=ctx, lo=lo, steps=steps)
        if _weight(work(case)) <= limit:
            return case


def _lengths(case):
    """context or prompt lengths, spread evenly from `lo` to `ctx`"""
    b, lo, hi = case['batch'], case['lo'], case['ctx']
    return np.array([hi] if b == 1 else [lo + (hi - lo) * i // (b - 1) for i in range(b)], np.int32)


class _Weights:
    """stands where a Hugging Face model stands: state_dict() under its names, made on the GPU from a seed"""

    def __init__(self, sh, seed):
        self.sh, self.g = sh, torch.Generator(device='cuda').manual_seed(seed)

    def _n(self, *shape, std, mean=0.0):
        return torch.randn(*shape, generator=self.g, device='cuda', dtype=torch.float32).mul_(std).add_(mean).half()

    def state_dict(self):
        sh, n = self.sh, self._n
        into = 0.02 / math.sqrt(2 * sh.L)
        sd = {'transformer.wte.weight': n(sh.N, sh.D, std=0.1), 'transformer.wpe.weight': n(sh.C, sh.D, std=0.05),
              'transformer.ln_f.weight': n(sh.D, std=0.1, mean=1.0), 'transformer.ln_f.bias': n(sh.D, std=0.02)}
        for l in range(sh.L):
            p = f'transformer.h.{l}.'
            for ln in ('ln_1', 'ln_2'):
                sd[p + ln + '.weight'], sd[p + ln + '.bias'] = n(sh.D, std=0.1, mean=1.0), n(sh.D, std=0.02)
            for name, i, o, std in (('attn.c_attn', sh.D, sh.J, 0.02), ('attn.c_proj', sh.D, sh.D, into),
                                    ('mlp.c_fc', sh.D, sh.F, 0.02), ('mlp.c_proj', sh.F, sh.D, into)):
                sd[p + name + '.weight'], sd[p + name + '.bias'] = n(i, o, std=std), n(o, std=0.02)
        return sd


def prepare(case, seed):
    sh, b, hi = SHAPES[case['model']], case['batch'], case['ctx']
    lens = np.random.RandomState(seed % (1 << 31)).permutation(_lengths(case)).astype(np.int32)
    ragged = case['lo'] != case['ctx']
    m = VestaGPT2(_Weights(sh, seed), batch=b, tmax=sh.C, per_sequence_t=ragged)
    g = torch.Generator(device='cuda').manual_seed(seed + 1)
    s = dict(case=case, m=m)
    if case['call'] == 'prefill':
        s['tokens'] = torch.randint(sh.N, (b, hi), generator=g, device='cuda').to(torch.int32).cpu().numpy()
        s['lengths'] = lens if ragged else None
        return s
    for cache in (m.keys, m.vals):
        cache[:, :, :hi].normal_(0.0, CACHE_STD, generator=g)
    s['t'] = torch.from_numpy(lens[:m.t.numel()].copy()).cuda()
    s['x'] = torch.randint(sh.N, (b,), generator=g, device='cuda').to(torch.int32)
    if case['call'] == 'host':
        s['first'] = s['x'].cpu().numpy()
        s['tokens'] = torch.empty(b, dtype=torch.int32).pin_memory()
        s['next'] = torch.empty(b, dtype=torch.float32).pin_memory()
        s['tokens_np'], s['next_np'] = s['tokens'].numpy(), s['next'].numpy()
    return s


def run(s):
    case, m = s['case'], s['m']
    hi, n = case['ctx'], case['steps']
    if case['call'] == 'prefill':
        m.prefill(s['tokens'], s['lengths'])
        return dict(x=m.x, t=m.t, keys=m.keys[:, :, :hi], vals=m.vals[:, :, :hi])
    m.t.copy_(s['t'])
    if case['call'] == 'host':
        s['tokens_np'][:] = s['first']
        chosen = []
        for _ in range(n):
            m.step_host(s['tokens'], s['next'])
            chosen.append(s['next_np'].astype(np.int32))
            s['tokens_np'][:] = chosen[-1]
        out = dict(chosen=np.stack(chosen))
    else:
        m.x.copy_(s['x'])
        m.step(n)
        out = dict(next=m.next())
    # the cache rows that the steps added (all rows from the shortest context on), the state and the last step's logits
    lo = case['lo']
    return dict(out, x=m.x, t=m.t, logits=m.logits(), keys=m.keys[:, :, lo:hi + n], vals=m.vals[:, :, lo:hi + n])


def _weight(w):
    return max(w['bytes'], w['flops'] / 50)


def work(case):
    sh, b, n = SHAPES[case['model']], case['batch'], case['steps']
    lens = _lengths(case).astype(np.int64)
    layer = sh.L * (sh.D * sh.J + sh.D * sh.D + 2 * sh.D * sh.F)            # weights of the layer contractions
    per_pos = sh.kv_bytes_per_pos()
    if case['call'] == 'prefill':
        pos, pairs = int(lens.sum()), int((lens * (lens + 1) // 2).sum())
        return dict(bytes=sh.weight_bytes() + pos * (per_pos + 4), flops=2 * layer * pos + 2 * sh.N * sh.D * b + 4 * sh.L * sh.D * pairs)
    attended = n * int((lens + 1).sum()) + b * n * (n - 1) // 2             # summed over the steps
    return dict(bytes=n * (sh.weight_bytes() + b * (sh.N * 4 + per_pos)) + per_pos * (attended - b * n),
                flops=2 * (layer + sh.N * sh.D) * b * n + 4 * sh.L * sh.D * attended)


def tolerance(case):
    # up to eight sequences the activations are multiplied at fp32 accuracy, what remains is the fp16 rounding of K and V;
    # above, the operands of the contractions are rounded to fp16 (2^-11), over all layers
    if case['call'] != 'prefill' and case['batch'] <= 8:
        return dict(rel=1e-3, differ=0.0)
    return dict(rel=3e-3, differ=0.0)
