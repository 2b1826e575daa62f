"""Forward passes as chains of kernels (csrc/pass.cu, csrc/pass_kernels.cuh, csrc/pass_few.cuh): the descriptor of a pass and the dense prompt
pass behind VestaGPT2.prefill."""
import ctypes
import weakref

import numpy as np
import torch

from .launch import STATUS_WHERE, lib, ok
from .lower import ZEROS

_PTRS = ('wte', 'wpe', 'ln1w', 'ln1b', 'qkvw', 'qkvb', 'ow', 'ob', 'ln2w', 'ln2b', 'fcw', 'fcb', 'pw', 'pb', 'lnfw', 'lnfb',
         'keys', 'vals', 'x', 't', 'prompt', 'plen', 'logits', 'next', 'bar')
WEIGHTS = _PTRS[:16]
VECTORS = ('ln1w', 'ln1b', 'qkvb', 'ob', 'ln2w', 'ln2b', 'fcb', 'pb', 'lnfw', 'lnfb')


class Desc(ctypes.Structure):
    """vesta_pass_desc (include/vesta_b200.h)"""
    _fields_ = [(n, ctypes.c_int) for n in ('L', 'D', 'H', 'F', 'N', 'tmax', 'cpos', 'rows', 'logit_rows', 'prompts', 'exact',
                                            't_stride', 'tstep', 'feedback', 'prompt_len')] + \
               [(n, ctypes.c_float) for n in ('eps', 'scale', 'gelu_a', 'gelu_b', 'gelu_c')] + \
               [(n, ctypes.c_void_p) for n in _PTRS]


def aligned(low, residue, roles, kept=()):
    """-> (`residue` as kernels that load 16 bytes at a time can read it, {name: (copy, original)}): the weights named by `roles`
    that do not start on a 16-byte boundary (views into a larger buffer) are copied, into the copies of `kept` where it has
    them. The table and the caches are read and written where they are: refused."""
    out, copies = dict(residue), {}
    for role in ('wte', 'keys', 'vals'):
        if residue[low.roles[role]].data_ptr() % 16:
            raise RuntimeError(f'{low.roles[role]} must start on a 16-byte boundary')
    for role in roles:
        name = low.roles[role]
        if name != ZEROS and residue[name].data_ptr() % 16:
            out[name] = kept[name][0].copy_(residue[name]) if name in kept else residue[name].clone()
            copies[name] = out[name], residue[name]
    return out, copies


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


def kernels_of_a_step(layers, few=False):
    """kernels that a decode step launches as a chain: seven per layer, the embedding with its norm, the logits, the end; of few
    sequences three per layer (the first makes the embedding), the last norm, the logits, the end"""
    return (3 if few else 7) * layers + 3


def tiles(desc, rows, logit_rows):
    """the tiles of the contractions of a pass over `rows` rows of which `logit_rows` want logits: for 'qkv', 'proj', 'fc', 'p2' and
    'logits' (features, rows, stages, parts of the fold, bytes of shared memory)"""
    out = (ctypes.c_int * 25)()
    ok(lib().vesta_pass_tiles(ctypes.byref(desc), rows, logit_rows, out))
    return {k: tuple(out[5 * i:5 * i + 5]) for i, k in enumerate(('qkv', 'proj', 'fc', 'p2', 'logits'))}


def create(desc, device, graph=False, ws=None):
    """-> (handle, workspace tensor). `ws`: the workspace of an earlier pass of the same sizes (every pass leaves it as it
    found it): a step that still runs on another stream then keeps its memory, and nothing has to be cleared or awaited"""
    if ws is None:
        n = ctypes.c_size_t()
        ok(lib().vesta_pass_workspace(ctypes.byref(desc), ctypes.byref(n)))
        ws = torch.zeros(n.value, dtype=torch.uint8, device=device)
        torch.cuda.current_stream(device).synchronize()
    h = ctypes.c_void_p()
    ok(lib().vesta_pass_create(ctypes.byref(desc), ctypes.c_void_p(ws.data_ptr()), int(graph), ctypes.byref(h)))
    return h, ws


def step_desc(kernel, residue, zeros):
    """the descriptor of a decode step over the tensors of `residue`"""
    low = kernel.lowered
    d, st = low.dims, low.dims['step']
    off = {n: kernel.S.data_ptr() + 4 * v[0] for n, v in low.scratch.items()}
    logit, nxt = list(off.values())
    return describe(low, residue, zeros, st['cpos'], rows=d['B'], logit_rows=d['B'], exact=st['exact'], t_stride=st['t_stride'],
                    tstep=st['tstep'], feedback=st['feedback'], prompt_len=st['prompt_len'], x=residue[low.roles['x']], t=residue[low.roles['t']],
                    prompt=residue['prompt'] if st['prompt_len'] else None, plen=residue['plen'] if st['prompt_len'] else None,
                    logits=logit, next=nxt, bar=kernel.bar)


def bind_step(kernel, residue, zeros, graph):
    """a decode step over the tensors of `residue` as a chain of kernels -> (handle for vesta_step_run, the pass that it owns, workspace)"""
    h, ws = create(step_desc(kernel, residue, zeros), kernel.device, graph, kernel._work)
    bound = ctypes.c_void_p()
    ok(lib().vesta_pass_bind(h, ctypes.byref(bound)))
    return bound, h, ws


def pack_step(kernel, residue):
    """the packed weights of a bound step of few sequences, made from the layers' matrices in `residue` instead of the bound ones"""
    low, (bound, zeros) = kernel.lowered, kernel._here
    names = [low.roles[r] for r in ('qkvw', 'ow', 'fcw', 'pw')]
    here, _ = aligned(low, {**bound, **{n: residue[n] for n in names}}, WEIGHTS[1:])
    h, _ = create(step_desc(kernel, here, zeros), kernel.device, ws=kernel._work)
    try:
        ok(lib().vesta_pass_pack(h, ctypes.c_void_p(torch.cuda.current_stream(kernel.device).cuda_stream)))
    finally:
        lib().vesta_pass_release(h)


class PromptPass:
    """Whole prompts as dense passes over up to `rows` (sequence, position) rows that write a model's caches, x and t: every
    row's K and V are written before any row attends, so a row sees the rows of its own sequence before it. Only the last
    position of a prompt wants logits."""

    def __init__(self, model, rows):
        dev, low = model.device, model.low
        lrows = min(rows, model.B)
        self.model, self.R = weakref.proxy(model), rows          # (the model owns the pass: no cycle, its memory is free when it goes)
        self.logits = torch.empty(lrows, low.dims['N'], dtype=torch.float32, device=dev)
        self.bar = torch.zeros(32, dtype=torch.int32, device=dev)
        self.zeros = torch.zeros(low.dims['zeros_len'], dtype=torch.float16, device=dev)
        R, self.copies = aligned(low, {**model.W, 'keys': model.keys, 'vals': model.vals}, WEIGHTS[1:])
        desc = describe(low, R, self.zeros, low.dims['step']['cpos'], rows=rows, logit_rows=lrows, prompts=model.B,
                        t_stride=int(model.t.numel() > 1), x=model.x, t=model.t, logits=self.logits, bar=self.bar)
        with torch.cuda.device(dev):
            self.h, self.ws = create(desc, dev)
        self._prompts = lib().vesta_pass_prompts
        self.desc = desc

    def run(self, tokens, lens):
        """tokens (B, P), lens (B,) int32 numpy: the caches, x and t of the model after the prompts"""
        tokens = np.ascontiguousarray(tokens, np.int32)
        for copy, original in self.copies.values():
            copy.copy_(original)
        dev, status = self.model.device, ctypes.c_uint()
        at = tokens.__array_interface__['data'][0], tokens.shape[1], lens.__array_interface__['data'][0], ctypes.byref(status)
        if torch.cuda.current_device() == dev.index:
            ok(self._prompts(self.h, torch.cuda.current_stream(dev).cuda_stream, *at))
        else:
            with torch.cuda.device(dev):
                ok(self._prompts(self.h, torch.cuda.current_stream(dev).cuda_stream, *at))
        v = status.value
        if v:
            self.bar.zero_()
            self.model.reset()
            raise RuntimeError(f'prefill gave up: {STATUS_WHERE.get(v & 0xff00, hex(v & 0xffff))}')

    def __del__(self):
        try:
            if getattr(self, 'h', None):
                lib().vesta_pass_release(self.h)
        except Exception:
            pass
