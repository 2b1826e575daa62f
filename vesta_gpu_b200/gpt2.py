"""The decode-step program on the GPU: Hugging Face style weights as residue, a step as one persistent kernel (few
sequences) or as a chain of kernels, prompts as dense passes of the same chain.

    m = VestaGPT2(hf, dtype='f16', batch=8, tmax=1024)
    m.reset(); m.x.copy_(tok); m.t.fill_(p); m.step()     # one decode step
    m.logits(), m.next()                                    # views, no sync

Same surface as the reference binding (vesta/gpt2.py:18-55): `gpt2_weights`, and `VestaGPT2`
with `W, B, tmax, keys, vals, x, t, low, k, weight_bytes, reset, step, logits, next, kv_bytes`.
With feedback on, each step writes its chosen token into x and advances t, so generation is
back-to-back launches with nothing from the host in between. The sizes (layers, width, heads,
MLP width, vocabulary) are read from the weights instead of being fixed to GPT-2 small
(vesta/gpt2.py:16), so an XL-shaped model runs through the same code.
"""
import torch

from . import PROGRAMS
from .launch import Kernel, TORCH_DT
from .lower import lower
from .passes import PromptPass
from .program_text import decode_program
from .shapes import Shape

E_HEAD = 64


def gpt2_weights(hf):
    """state_dict under Hugging Face names -> residues of the step program, per-layer tensors stacked on l"""
    sd = hf.state_dict()
    L = 0
    while f'transformer.h.{L}.ln_1.weight' in sd:
        L += 1
    st = lambda n: torch.stack([sd[f'transformer.h.{l}.{n}'] for l in range(L)])
    return dict(wte=sd['transformer.wte.weight'], wpe=sd['transformer.wpe.weight'],
                ln1w=st('ln_1.weight'), ln1b=st('ln_1.bias'), qkvw=st('attn.c_attn.weight'), qkvb=st('attn.c_attn.bias'),
                ow=st('attn.c_proj.weight'), ob=st('attn.c_proj.bias'), ln2w=st('ln_2.weight'), ln2b=st('ln_2.bias'),
                fcw=st('mlp.c_fc.weight'), fcb=st('mlp.c_fc.bias'), pw=st('mlp.c_proj.weight'), pb=st('mlp.c_proj.bias'),
                lnfw=sd['transformer.ln_f.weight'], lnfb=sd['transformer.ln_f.bias'])


def shape_of(W, heads=None):
    N, D = W['wte'].shape
    L, _, F = W['fcw'].shape
    H = heads or D // E_HEAD
    return Shape('model', L=L, D=D, H=H, E=D // H, F=F, N=N, C=W['wpe'].shape[0])


# rows per dense pass of prefill(): a pass that holds more rows fills the GPU better, up to where all SMs are busy in every kernel
PREFILL_ROWS = (128, 256, 512, 1024, 2048, 4096, 8192, 16384)


class VestaGPT2:
    def __init__(self, hf, dtype='f16', batch=1, tmax=1024, feedback=True, program=None, timing=False,
                 blocks_per_sm=None, per_sequence_t=False, device=None, prompt_len=0, slab_tiles=None, tune=None, without=()):
        """program: path of a .vst file; default: the step program for the sizes of the weights
        (identical to programs/gpt2.vst for GPT-2 small), `without` naming the shifts and biases it leaves out
        (program_text.ADDITIVE). Weights the program does not receive are not bound. per_sequence_t: every sequence keeps its
        own position t[b] (ragged batches); default one position for the whole batch as in the
        reference. prompt_len > 0 adds the buffers `prompt` (batch, prompt_len) and `plen` (batch,): the
        kernel then feeds prompt[b][t+1] while t + 1 < plen[b] and its own choice afterwards."""
        tdt = TORCH_DT[dtype]
        dev = torch.device('cuda', torch.cuda.current_device() if device is None else device)
        self.device = dev
        self.W = {k: v.detach().to(dev, tdt).contiguous() for k, v in gpt2_weights(hf).items()}
        self.shape = shape_of(self.W)
        sh = self.shape
        self.B, self.tmax = batch, tmax
        self.keys = torch.zeros(batch, sh.L, tmax, sh.H, sh.E, device=dev, dtype=tdt)
        self.vals = torch.zeros_like(self.keys)
        self.x = torch.zeros(batch, dtype=torch.int32, device=dev)
        self.t = torch.zeros(batch if per_sequence_t else 1, dtype=torch.int32, device=dev)
        R = {'x': self.x, 't': self.t, **self.W, 'keys': self.keys, 'vals': self.vals}
        if prompt_len:
            self.prompt = torch.zeros(batch, prompt_len, dtype=torch.int32, device=dev)
            self.plen = torch.zeros(batch, dtype=torch.int32, device=dev)
        names = {torch.int32: 'i32', torch.float16: 'f16', torch.float32: 'f32'}
        spec = {n: (((batch,) if per_sequence_t else ()), 'i32') if n == 't' else (tuple(v.shape), names[v.dtype])
                for n, v in R.items() if n not in ('prompt', 'plen')}
        if program is None:
            text = decode_program(sh, without=tuple(without))
        else:
            text = open(program, encoding='utf-8').read()
        from .lower import recognise
        recv = set(recognise(text)[2])
        self.W = {n: v for n, v in self.W.items() if n in recv}
        R = {n: v for n, v in R.items() if n in recv}
        spec = {n: v for n, v in spec.items() if n in recv}
        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        per_token = ('x', 'keys', 'vals') + (('t',) if per_sequence_t else ())
        self.low = lower(text, spec, axis_max={'s': tmax}, batch=batch, per_token=per_token,
                         outputs=('logit', 'next'), feedback={'x': 'next', 't': 1} if feedback else None,
                         timing=timing, grid=sms, prompt_len=prompt_len if feedback else 0, slab_tiles=slab_tiles, tune=tune)
        self._prefill_engines = {}
        self.k = Kernel(self.low, device=dev.index, blocks_per_sm=blocks_per_sm)
        if prompt_len and feedback:
            R = dict(R, prompt=self.prompt, plen=self.plen)
        self.k.bind(R)
        self.weight_bytes = sum(v.numel() * v.element_size() for n, v in self.W.items() if n != 'wpe') \
            + sh.D * self.W['wpe'].element_size()

    def reset(self):
        self.keys.zero_(); self.vals.zero_(); self.t.zero_()

    def step(self, steps=1):
        self.k.launch(steps)

    def step_host(self, tokens_host, next_host):
        """one step for a host-side loop: tokens_host (pinned int32 [batch]) becomes x, the chosen tokens (the
        `next` values, float32 [batch] as in the reference's scratch) land in next_host (pinned); returns when
        they have"""
        nv = self.__dict__.get('_next_view')
        if nv is None:
            nv = self._next_view = self.next()              # (a view of the scratch area: made once, a host loop calls this per step)
        self.k.step_host(self.x, tokens_host, nv, next_host)

    def prefill(self, tokens, lengths=None, rows=None):
        """consume whole prompts as dense passes: all prompt positions of all sequences are cut into passes of at most `rows`
        (sequence, position) rows (default: the smallest of PREFILL_ROWS that holds them all, or its largest), see
        passes.PromptPass. On return the cache holds every prompt position, x the first generated token
        of every sequence and t its position (= its prompt length). tokens: int array (batch, P); lengths: (batch,) or
        None for P everywhere (lengths that differ need per_sequence_t=True).
        The reference feeds the prompt one position per step (bench/g0_bench.py:172-173); prefill_stepwise does the same
        on the device."""
        import numpy as np
        tokens = np.asarray(tokens)
        B, P = tokens.shape
        if B != self.B:
            raise ValueError('prefill needs one prompt per sequence of the batch')
        if lengths is None:
            lens, low, high, total = np.full(B, P, np.int32), P, P, B * P
        else:
            lens = np.ascontiguousarray(lengths, np.int32)
            if lens.shape != (B,):
                raise ValueError('one prompt length per sequence')
            low, high, total = int(lens.min()), int(lens.max()), int(lens.sum())
        if low < 1 or high > P or high > self.tmax:
            raise ValueError('prompt lengths must lie in 1..P and fit the cache')
        if self.t.numel() == 1 and low != high:
            raise ValueError('prompts of different lengths need per_sequence_t=True')
        rows = int(rows or next((r for r in PREFILL_ROWS if total <= r), PREFILL_ROWS[-1]))
        eng = self._prefill_engines.get(rows)
        if eng is None:
            eng = self._prefill_engines[rows] = PromptPass(self, rows)
        eng.run(tokens, lens)
        if hasattr(self, 'prompt'):
            buf = np.zeros(tuple(self.prompt.shape), np.int32)
            w = min(P, buf.shape[1])
            buf[:, :w] = tokens[:, :w]
            self.prompt.copy_(torch.from_numpy(buf)); self.plen.copy_(torch.from_numpy(np.minimum(lens, buf.shape[1]).astype(np.int32)))

    def prefill_stepwise(self, tokens, lengths=None):
        """consume whole prompts one position per step, fed on the device (needs prompt_len >= the longest prompt and
        per_sequence_t when the lengths differ): the prompts go to the device once, then the kernel feeds itself, several
        steps per launch, until every prompt has been read; sequences shorter than the longest start late (negative
        positions) so that all of them end together. On return x holds the first generated token of every sequence and
        t its position. tokens: int array (batch, P), lengths: (batch,) or None for P everywhere."""
        import numpy as np
        tokens = np.asarray(tokens)
        B, P = tokens.shape
        if not hasattr(self, 'prompt') or B != self.B or P > self.prompt.shape[1]:
            raise ValueError('prefill_stepwise needs a model built with prompt_len >= the prompt length and the same batch')
        lens = np.full(B, P, np.int32) if lengths is None else np.asarray(lengths, np.int32)
        if lens.min() < 1 or lens.max() > P:
            raise ValueError('prompt lengths must lie in 1..P')
        pmax = int(lens.max())
        if self.t.numel() == 1 and lens.min() != pmax:
            raise ValueError('prompts of different lengths need per_sequence_t=True')
        buf = np.zeros(tuple(self.prompt.shape), np.int32)
        buf[:, :P] = tokens
        self.reset()
        self.prompt.copy_(torch.from_numpy(buf)); self.plen.copy_(torch.from_numpy(lens))
        start = (lens - pmax).astype(np.int32)
        self.t.copy_(torch.from_numpy(start[:self.t.numel()]))
        self.x.copy_(torch.from_numpy(np.where(start == 0, tokens[:, 0], 0).astype(np.int32)))
        self.k.launch(pmax)

    def state(self):
        """the decode state (cache, tokens, positions) as CPU tensors, for load_state() on a model of the same
        shape, batch and tmax: generation then continues where it stood"""
        return {'keys': self.keys.cpu(), 'vals': self.vals.cpu(), 'x': self.x.cpu(), 't': self.t.cpu()}

    def load_state(self, st):
        for name in ('keys', 'vals', 'x', 't'):
            dst, src = getattr(self, name), st[name]
            if tuple(dst.shape) != tuple(src.shape) or dst.dtype != src.dtype:
                raise ValueError(f'state[{name!r}] is {tuple(src.shape)} {src.dtype}, the model holds {tuple(dst.shape)} {dst.dtype}')
            dst.copy_(src)

    def logits(self):
        return self.k.view('logit')

    def next(self):
        return self.k.view('next')

    def kv_bytes(self, n_ctx):
        sh = self.shape
        return 2 * sh.L * self.B * n_ctx * sh.D * self.keys.element_size()


DEFAULT_PROGRAM = PROGRAMS / 'gpt2.vst'
