"""Forward passes as chains of kernels (csrc/pass.cu, csrc/pass_kernels.cuh): the descriptor of a pass and the dense prompt
pass behind VestaGPT2.prefill."""
import ctypes

import numpy as np
import torch

from .launch import STATUS_WHERE, lib, ok
from .lower import Lowered, ZEROS

_PTRS = ('wte', 'wpe', 'ln1w', 'ln1b', 'qkvw', 'qkvb', 'ow', 'ob', 'ln2w', 'ln2b', 'fcw', 'fcb', 'pw', 'pb', 'lnfw', 'lnfb',
         'keys', 'vals', 'x', 't', 'seq', 'prompt', 'plen', 'tiles', 'want', 'dst', 'x_out', 'logits', 'next', 'bar')
WEIGHTS = _PTRS[:16]


class Desc(ctypes.Structure):
    """vesta_pass_desc (include/vesta_b200.h)"""
    _fields_ = [(n, ctypes.c_int) for n in ('L', 'D', 'H', 'F', 'N', 'tmax', 'cpos', 'rows', 'logit_rows', 'exact',
                                            't_stride', 'tstep', 'feedback', 'prompt_len')] + \
               [(n, ctypes.c_float) for n in ('eps', 'scale', 'gelu_a', 'gelu_b', 'gelu_c')] + \
               [(n, ctypes.c_void_p) for n in _PTRS]


def describe(low, residue, zeros, cpos, **kw):
    """the descriptor of a pass over the program `low` (lower.Lowered) with the tensors of `residue`; kw: further fields,
    tensors or numbers"""
    d = low.dims
    desc = Desc(L=d['L'], D=d['D'], H=d['H'], F=d['F'], N=d['N'], tmax=d['tmax'], cpos=cpos, eps=d['eps'], scale=d['scale'],
                gelu_a=d['gelu'][0], gelu_b=d['gelu'][1], gelu_c=d['gelu'][2])
    for role in WEIGHTS + ('keys', 'vals'):
        name = low.roles[role]
        setattr(desc, role, (zeros if name == ZEROS else residue[name]).data_ptr())
    for k, v in kw.items():
        if v is not None:
            setattr(desc, k, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    return desc


def create(desc, device, graph=False):
    """-> (handle, workspace tensor)"""
    n = ctypes.c_size_t()
    ok(lib().vesta_pass_workspace(ctypes.byref(desc), ctypes.byref(n)))
    ws = torch.zeros(n.value, dtype=torch.uint8, device=device)
    h = ctypes.c_void_p()
    torch.cuda.current_stream(device).synchronize() if graph else None
    ok(lib().vesta_pass_create(ctypes.byref(desc), ctypes.c_void_p(ws.data_ptr()), int(graph), ctypes.byref(h)))
    return h, ws


def bind_step(kernel, residue, zeros):
    """a decode step over the tensors of `residue` as a chain of kernels -> (handle for vesta_step_run, workspace)"""
    low = kernel.lowered
    d, st = low.dims, low.dims['step']
    off = {n: kernel.S.data_ptr() + 4 * v[0] for n, v in low.scratch.items()}
    logit, nxt = list(off.values())
    desc = describe(low, residue, zeros, st['cpos'], rows=d['B'], logit_rows=d['B'], exact=st['exact'], t_stride=st['t_stride'],
                    tstep=st['tstep'], feedback=st['feedback'], prompt_len=st['prompt_len'], x=residue[low.roles['x']], t=residue[low.roles['t']],
                    prompt=residue['prompt'] if st['prompt_len'] else None, plen=residue['plen'] if st['prompt_len'] else None,
                    logits=logit, next=nxt, bar=kernel.bar)
    h, ws = create(desc, kernel.device, graph=True)
    bound = ctypes.c_void_p()
    ok(lib().vesta_pass_bind(h, ctypes.byref(bound)))
    return bound, ws


class PromptPass:
    """Whole prompts as dense passes over up to `rows` (sequence, position) rows that write a model's caches: every row's
    K and V are written before any row attends, so a row sees the rows of its own sequence before it. Only the last
    position of a prompt wants logits."""

    TILE = 64                                     # rows of one sequence per attention block (csrc/pass_kernels.cuh)

    def __init__(self, model, rows):
        dev = model.device
        self.model, self.R, self.LR = model, rows, min(rows, model.B)
        d = model.low.dims
        self.nt = rows // self.TILE + min(rows, model.B) + 1
        self.off = np.cumsum([0, rows, rows, rows, 4 * self.nt, self.LR, self.LR])
        self.meta = torch.zeros(int(self.off[-1]), dtype=torch.int32, device=dev)
        self.host = []                            # pinned copies of the metadata, one per launch of a call
        part = [self.meta[a:] for a in self.off[:-1]]
        self.first = torch.zeros(model.B, dtype=torch.int32, device=dev)
        self.logits = torch.empty(self.LR, d['N'], dtype=torch.float32, device=dev)
        self.bar = torch.zeros(32, dtype=torch.int32, device=dev)
        self.zeros = torch.zeros(d['zeros_len'], dtype=torch.float16, device=dev)
        R = {**model.W, 'keys': model.keys, 'vals': model.vals}
        self.desc = describe(model.low, R, self.zeros, model.W[model.low.roles['wpe']].shape[0], rows=rows, logit_rows=self.LR, t_stride=1,
                             x=part[0], t=part[1], seq=part[2], tiles=part[3], want=part[4], dst=part[5], x_out=self.first,
                             logits=self.logits, bar=self.bar)
        with torch.cuda.device(dev):
            self.h, self.ws = create(self.desc, dev)
        self.low = Lowered(src='', params=[], scratch={}, scratch_floats=0, shared_bytes=0, barriers_per_launch=0, grid=model.low.grid,
                           plan=[('prompt rows', 'one kernel per norm, contraction and attention of a layer, tcgen05 contractions')],
                           dims=dict(d, B=rows, kernel='pass', tc=True, tcl=True), roles=model.low.roles)

    def run(self, tokens, lens):
        """tokens (B, P), lens (B,) numpy -> int32 tensor (B,) on the device: the token chosen after every prompt"""
        B, R, T = tokens.shape[0], self.R, self.TILE
        ends = np.cumsum(lens)
        total = int(ends[-1])
        starts = ends - lens
        seqs = np.repeat(np.arange(B, dtype=np.int32), lens)
        pos = (np.arange(total, dtype=np.int32) - np.repeat(starts.astype(np.int32), lens))
        tok = tokens[seqs, pos]
        stream = ctypes.c_void_p(torch.cuda.current_stream(self.model.device).cuda_stream)
        for c, i in enumerate(range(0, total, R)):
            n = min(R, total - i)
            if c == len(self.host):
                self.host.append(torch.zeros(self.meta.numel(), dtype=torch.int32).pin_memory())
            m, off = self.host[c].numpy(), self.off
            m[off[0]:off[0] + n], m[off[1]:off[1] + n], m[off[2]:off[2] + n] = tok[i:i + n], pos[i:i + n], seqs[i:i + n]
            # runs of at most TILE rows of one sequence; the ones that see most positions first
            here = np.flatnonzero((ends > i) & (starts < i + n))
            lo, hi = np.maximum(starts[here], i), np.minimum(ends[here], i + n)
            k = -(-(hi - lo) // T)
            which = np.repeat(np.arange(len(here)), k)
            piece = np.arange(len(which)) - np.repeat(np.cumsum(k) - k, k)
            r0 = lo[which] + piece * T
            rows = np.minimum(T, hi[which] - r0)
            p0 = r0 - starts[here][which]
            order = np.argsort(-(p0 + rows), kind='stable')
            tl = np.stack([r0 - i, rows, here[which], p0], 1)[order]
            m[off[3]:off[3] + 4 * len(tl)] = tl.reshape(-1)
            done = here[ends[here] <= i + n]
            m[off[4]:off[4] + len(done)], m[off[5]:off[5] + len(done)] = ends[done] - 1 - i, done
            self.meta.copy_(self.host[c], non_blocking=True)
            ok(lib().vesta_pass_run(self.h, stream, n, len(done), len(tl)))
        v = int(self.bar[0].item())
        if v:
            self.bar.zero_()
            raise RuntimeError(f'prefill gave up: {STATUS_WHERE.get(v & 0xff00, hex(v & 0xffff))}')
        return self.first

    def __del__(self):
        try:
            if getattr(self, 'h', None):
                lib().vesta_pass_release(self.h)
        except Exception:
            pass
