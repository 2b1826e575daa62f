"""Passes as chains of kernels (csrc/pass.cu) at the edges of their tiles and dispatch rules, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import TIGHT, MARGIN
from test_gpu_parity import model

pytestmark = pytest.mark.gpu


def shape(name, **kw):
    """two or three narrow layers with room for 400 positions"""
    from vesta_gpu_b200.shapes import Shape
    return Shape(name, **dict(dict(L=2, D=192, H=3, E=64, F=320, N=333, C=400), **kw))


def seeded(m, sh, ctx, seed):
    """caches of `ctx[b]` positions per sequence -> the oracle's copies"""
    from vesta_gpu_b200.synth import make_cache
    out = []
    m.reset()
    for b, c in enumerate(ctx):
        k0, v0 = make_cache(sh, seed + b, int(c))
        ck, cv = np.zeros((sh.L, m.tmax, sh.H, sh.E), np.float16), np.zeros((sh.L, m.tmax, sh.H, sh.E), np.float16)
        ck[:, :c] = k0
        cv[:, :c] = v0
        out.append((ck, cv))
        m.keys[b, :, :c].copy_(torch.from_numpy(k0))
        m.vals[b, :, :c].copy_(torch.from_numpy(v0))
    return out


@pytest.mark.parametrize('batch,kw', [
    (9, {}), (16, {}), (17, {}),                      # operands at fp32 accuracy up to 16 rows; two blocks per (row, head) in the attention
    (64, {}), (65, {}),                               # edges of a tile of rows
    (130, {}),                                        # more (row, head) pairs than blocks in flight: one block each
    (200, {}),                                        # ... and shallow rings
    (9, dict(D=320, H=5, F=1296)),                    # folds of five blocks, the last block of the second one ragged
    (16, dict(D=1216, H=19, F=64)),                   # a fold of 19 blocks, fp16 operands at 16 rows
    (8, dict(L=1, D=1280, H=20)),                     # 160 (sequence, head) pairs at eight sequences: a chain, not the persistent kernel
    (3, dict(L=1, D=1344, H=21)),                     # three sequences of a wide shape: the same
    # every shape of the attention past the ends of its rings: eight warps with three stages, in clusters of two and alone, also of wide rows,
    (11, dict(L=1, D=640, H=10, C=1200)), (80, dict(C=1200)), (11, dict(L=1, D=1536, H=24, F=64, C=1200)),
    # with two; four warps with four stages, in clusters of two and alone, and with two
    (13, dict(L=1, D=1536, H=24, F=64, C=1200)), (9, dict(C=1200)), (16, dict(D=1216, H=19, F=64, C=1200)), (130, dict(C=1200)), (200, dict(C=1200)),
])
def test_step_as_a_chain(batch, kw):
    """ragged decode steps over seeded caches, contexts from none to nearly all of the cache"""
    from oracle import gpt2_numpy as O
    sh, steps = shape('chain', **kw), 2
    m, hf = model(sh, 17, 'rich', batch, sh.C, per_sequence_t=True)
    assert m.low.dims['chain']
    W = O.upcast(hf.weights)
    ctx = np.array([(37 * b) % (sh.C - 10) for b in range(batch)], np.int32)
    ctx[:4] = (sh.C - 11, 0, 63, 64)[:batch]
    caches = seeded(m, sh, ctx, 900)
    x = np.array([(b * 31 + 5) % sh.N for b in range(batch)], np.int32)
    m.t.copy_(torch.from_numpy(ctx))
    m.x.copy_(torch.from_numpy(x))
    some = sorted(set(range(min(5, batch))) | set(range(5, batch, max(1, batch // 12))) | {batch - 1})
    for s in range(steps):
        m.step()
        lg, nx = m.logits().cpu().numpy(), m.x.cpu().numpy()
        for b in some:
            ref, rn = O.step(sh, W, *caches[b], int(x[b]), int(ctx[b]) + s)
            assert np.abs(lg[b] - ref).max() < TIGHT * (1 if batch <= 16 and sh.D <= 1024 or batch <= 8 else 2), (s, b)
            if O.margin(ref) > MARGIN:
                assert int(nx[b]) == rn
        x = nx
    for b in some:
        c = int(ctx[b])
        assert np.abs(m.keys[b, :, c:c + steps].float().cpu().numpy() - caches[b][0][:, c:c + steps].astype(np.float32)).max() <= 4e-3
    m.k.check()


@pytest.mark.parametrize('batch,kw', [
    (2, {}), (3, {}), (4, {}),                        # heads and remainders side by side; 4 and 2 blocks per sequence in the attention
    (2, dict(D=64, H=1, F=16)),                       # fewer units of the fold, and of the outputs, than warps
    (4, dict(D=320, H=5, F=1296)),                    # ten pairs of units for eight warps
    (2, dict(L=1, D=1024, H=16, F=4096)), (4, dict(L=1, D=1024, H=16, F=2384)),   # two tiles per block; 149 tiles, the last block has one
    (3, dict(L=1, D=832, H=13, F=2384)),
])
def test_step_of_few_sequences(batch, kw, monkeypatch):
    """three kernels per layer from packed weights: ragged steps over seeded caches against the oracle; of two sequences the same bits
    twice"""
    from oracle import gpt2_numpy as O
    monkeypatch.setattr('vesta_gpu_b200.lower.few_pays', lambda D, F: True)          # (also where the persistent kernel is faster)
    sh, steps = shape('few', **kw), 2
    m, hf = model(sh, 17, 'rich', batch, sh.C, per_sequence_t=True)
    assert m.k.few and not m.k.chain
    W = O.upcast(hf.weights)
    ctx = np.array((389, 0, 63, 64, 255, 256, 257, 18)[:batch], np.int32)
    first = np.array([(b * 31 + 5) % sh.N for b in range(batch)], np.int32)
    runs = []
    for _ in range(2):
        caches, x = seeded(m, sh, ctx, 900), first
        m.t.copy_(torch.from_numpy(ctx))
        m.x.copy_(torch.from_numpy(x))
        for s in range(steps):
            m.step()
            lg, nx = m.logits().cpu().numpy(), m.x.cpu().numpy()
            for b in range(batch):
                ref, rn = O.step(sh, W, *caches[b], int(x[b]), int(ctx[b]) + s)
                assert np.abs(lg[b] - ref).max() < TIGHT, (s, b)
                assert O.margin(ref) <= MARGIN or int(nx[b]) == rn
            x = nx
        for b in range(batch):
            c = int(ctx[b])
            assert np.abs(m.keys[b, :, c:c + steps].float().cpu().numpy() - caches[b][0][:, c:c + steps].astype(np.float32)).max() <= 4e-3
        runs.append((m.logits().clone(), m.keys.clone(), m.vals.clone()))
    assert batch > 2 or all(torch.equal(a, b) for a, b in zip(*runs))
    m.k.check()


@pytest.mark.parametrize('ctx', [(1189, 1023), (511, 1024), (1189, 512, -1), (257, 513, 767), (1189, -1, 511, 1040), (255, 256, 768, 1023)])
def test_steps_of_few_sequences_past_the_ends_of_their_rings(ctx):
    """contexts that take a warp's ring of two stages (of 512 positions between them with two sequences, 256 with three and four) round more
    than once, the current position in the first round of a stage and in later ones, a sequence that starts a step later; against the oracle
    and the persistent kernel"""
    from oracle import gpt2_numpy as O
    sh, batch = shape('rings', C=1200), len(ctx)
    m, hf = model(sh, 17, 'rich', batch, sh.C, per_sequence_t=True)
    p, _ = model(sh, 17, 'rich', batch, sh.C, per_sequence_t=True, tune=dict(wait_ns=500_000_000))
    assert m.k.few and not p.k.graphs
    W = O.upcast(hf.weights)
    caches = seeded(m, sh, np.maximum(ctx, 0), 900)
    seeded(p, sh, np.maximum(ctx, 0), 900)
    x = np.array([(b * 31 + 5) % sh.N for b in range(batch)], np.int32)
    for s in range(2):
        for k in (m, p):
            k.t.copy_(torch.tensor([c + s for c in ctx], dtype=torch.int32))
            k.x.copy_(torch.from_numpy(x))
            k.step()
            k.k.check()
        lg, other, nx = m.logits().cpu().numpy(), p.logits().cpu().numpy(), m.next().cpu().numpy()
        for b in range(batch):
            if ctx[b] + s < 0:
                assert not m.keys[b].any() and not m.vals[b].any()
                continue
            ref, rn = O.step(sh, W, *caches[b], int(x[b]), ctx[b] + s)
            assert np.abs(lg[b] - ref).max() < TIGHT and np.abs(lg[b] - other[b]).max() < TIGHT, (s, b)
            assert O.margin(ref) <= MARGIN or int(nx[b]) == rn
            x[b] = rn
    for b in range(batch):
        for got, ref in ((m.keys, caches[b][0]), (m.vals, caches[b][1])):
            assert np.abs(got[b].float().cpu().numpy() - ref.astype(np.float32)).max() <= 4e-3, b


def test_equal_prompts_are_as_exact_in_every_batch():
    """GPT-2 small, the same sixteen tokens alone and as two to eight equal rows, in the persistent kernel and in the chain of few sequences:
    every row against the same arithmetic in 64 bits with K and V rounded to fp16. What is left are K and V that round the other way, as
    their sums differ from the exact ones in the last bits of fp32: over twelve prompts the persistent kernel's logits are at most 1.5 to
    1.8e-4 off (root mean square 2e-5), the chain's at most 0.95 to 1.14e-4 (1.7e-5), so two batches differ by up to 3e-4"""
    import math
    from vesta_gpu_b200.gpt2 import VestaGPT2
    from vesta_gpu_b200.shapes import GPT2_SMALL as sh
    from vesta_gpu_b200.synth import SynthGPT2, make_prompts
    P = 16
    hf = SynthGPT2(sh, 0, 'baseline')
    W = {n: torch.from_numpy(np.asarray(w)).cuda().double() for n, w in hf.weights.items()}
    prompts = [make_prompts(sh, 1, P, seed=s)[0] for s in (5, 6, 7)]
    toks = torch.from_numpy(np.stack(prompts).astype(np.int64)).cuda()

    def norm(z, w, b):
        m = z.mean(-1, keepdim=True)
        return (z - m) / torch.sqrt(((z - m) ** 2).mean(-1, keepdim=True) + 1e-5) * w + b
    heads = lambda a: a.view(len(prompts), P, sh.H, sh.E).transpose(1, 2)
    z = W['wte'][toks] + W['wpe'][:P]
    later = torch.full((P, P), -math.inf, device='cuda', dtype=torch.float64).triu(1)
    for l in range(sh.L):
        q, k, v = (norm(z, W['ln1w'][l], W['ln1b'][l]) @ W['qkvw'][l] + W['qkvb'][l]).split(sh.D, -1)
        w = torch.softmax(heads(q) @ heads(k.half().double()).transpose(-1, -2) / 8 + later, -1)
        z = z + (w @ heads(v.half().double())).transpose(1, 2).reshape(len(prompts), P, sh.D) @ W['ow'][l] + W['ob'][l]
        u = norm(z, W['ln2w'][l], W['ln2b'][l]) @ W['fcw'][l] + W['fcb'][l]
        z = z + (0.5 * u * (1 + torch.tanh(0.7978845608028654 * (u + 0.044715 * u ** 3)))) @ W['pw'][l] + W['pb'][l]
    exact = norm(z[:, -1], W['lnfw'], W['lnfb']) @ W['wte'].T
    for B in (1, 2, 3, 4, 5, 8):
        m = VestaGPT2(hf, batch=B, tmax=P + 1)
        assert m.k.few == (2 <= B <= 4) and not m.k.chain
        for i, prompt in enumerate(prompts):
            m.reset()
            for t in range(P):
                m.x.fill_(int(prompt[t]))
                m.step()
            off = m.logits().double() - exact[i]
            assert off.abs().max() < 3e-4 and off.square().mean().sqrt() < 4e-5, (B, i)     # (twice and less what was seen)
        m.k.check()


def test_a_good_step_of_few_sequences_runs_after_a_refused_one():
    """a position outside the cache: nothing is published; the status stays, the next step runs; after an abort flag none does"""
    sh = shape('refused few')
    m, _ = model(sh, 3, 'rich', 3, 100, per_sequence_t=True)
    m.reset()
    m.t.fill_(7)
    m.step()
    logits, keys = m.logits().clone(), m.keys.clone()
    m.t[1] = 100
    x, t = m.x.clone(), m.t.clone()
    m.step(2)
    assert torch.equal(m.logits(), logits) and torch.equal(m.keys, keys) and torch.equal(m.x, x) and torch.equal(m.t, t)
    assert 'out of range' in str(m.k.status())
    m.t.fill_(8)
    m.step()
    assert (m.t == 9).all() and not torch.equal(m.keys, keys)
    m.k.bar[2].fill_(1)
    m.step()
    assert (m.t == 9).all()
    m.k.clear_status()
    m.step()
    assert (m.t == 10).all()
    m.k.check()


def test_refused_step_stays_refused():
    """a position outside the cache, then the abort flag alone: nothing is published, later steps are refused until the status is cleared"""
    sh = shape('refused')
    m, _ = model(sh, 3, 'rich', 12, 100, per_sequence_t=True)
    for spoil in (lambda: m.t.fill_(100), lambda: m.k.bar[2].fill_(1)):
        m.reset()
        m.t.fill_(7)
        spoil()
        m.step(2)
        m.t.fill_(7)
        m.x.fill_(1)
        keys = m.keys.clone()
        m.step(2)
        assert (m.t == 7).all() and (m.x == 1).all() and torch.equal(keys, m.keys)
        with pytest.raises(RuntimeError):
            m.k.check()
        m.k.clear_status()
        m.step(2)
        m.k.check()
        assert (m.t == 9).all()


@pytest.mark.parametrize('lens,rows,kw,divisor', [
    ((9, 3, 1), 5, {}, 8),                                      # passes of five rows: less than one product of 16
    ((127, 128, 129, 1, 255, 257, 16, 384), None, {}, 8),       # edges of the attention's runs
    ((127, 128, 129, 1, 255, 257, 16, 384), 256, {}, 8),        # prompts that several passes read
    ((77,), None, dict(D=320, H=5, F=1296), 8),                 # one prompt, folds of five blocks, a ragged one behind
    ((200, 131), None, {}, 7),                                  # scores divided by what is not a power of two
    (tuple(range(60, 380, 10)), None, dict(D=768, H=12, F=832), 8),   # 6,880 rows: norms by warps, pairs of blocks, several tiles per block
])
def test_prompts_as_a_pass(lens, rows, kw, divisor, tmp_path):
    """first token, keys and values of every prompt position and zeros behind them"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.program_text import decode_program
    sh, batch, lens = shape('prompts', **kw), len(lens), np.array(lens, np.int32)
    more = {}
    if divisor != 8:
        text = decode_program(sh)
        assert text.count('/ 8\n') == 1
        (tmp_path / 'p.vst').write_text(text.replace('/ 8\n', f'/ {divisor}\n'))
        more = dict(program=str(tmp_path / 'p.vst'))
    m, hf = model(sh, 23, 'rich', batch, sh.C, per_sequence_t=True, **more)
    W = O.upcast(hf.weights)
    toks = np.random.RandomState(5).randint(0, sh.N, (batch, int(lens.max()))).astype(np.int32)
    m.keys.fill_(1.0)
    m.vals.fill_(1.0)
    m.prefill(toks, lens, rows=rows)
    assert m.t.cpu().numpy().tolist() == lens.tolist()
    for i in range(batch):
        assert not m.keys[i, :, lens[i]:].any() and not m.vals[i, :, lens[i]:].any()
    first = m.x.cpu().numpy()
    ref_w = dict(W)
    if divisor != 8:                                            # the oracle divides by 8
        ref_w['qkvw'], ref_w['qkvb'] = W['qkvw'].copy(), W['qkvb'].copy()
        ref_w['qkvw'][:, :, :sh.D] *= np.float32(8 / divisor)
        ref_w['qkvb'][:, :sh.D] *= np.float32(8 / divisor)
    for i in range(batch) if batch <= 8 else (0, 17, batch - 1):
        ck, cv = O.new_cache(sh, int(lens[i]))
        for p in range(int(lens[i])):
            lg, nx = O.step(sh, ref_w, ck, cv, int(toks[i, p]), p)
        for got, ref in ((m.keys, ck), (m.vals, cv)):
            assert np.abs(got[i, :, :lens[i]].float().cpu().numpy() - ref.astype(np.float32)).max() <= 4e-3, i
        if O.margin(lg) > MARGIN:
            assert int(first[i]) == nx


def overflowing(sh, seed):
    """weights of a one-layer model in which token 1 drives one GELU output past fp16 and no other token does: the first FC
    column points where token 1's normalised embedding does, and its row of the MLP projection is zero -> (model, its weights)"""
    from vesta_gpu_b200.synth import SynthGPT2, make_weights
    w = make_weights(sh, seed, 'rich')
    w['wte'][1] *= 20
    w['fcw'][0, :, 0] = np.sign(w['wte'][1].astype(np.float32)) * 700
    w['pw'][0, 0] = 0
    return SynthGPT2(sh, seed, weights=w), w


@pytest.mark.parametrize('batch', [12, 20])
def test_a_row_that_overflows_leaves_its_neighbours_alone(batch):
    """an MLP width that is no multiple of 64: the last fold block of the MLP projection ends inside a row's padding, so an
    infinity (or, as head and remainder, a NaN) in one sequence stays in that sequence; steps and prompts"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.gpt2 import VestaGPT2
    sh = shape('ragged', L=1, F=80)
    hf, w = overflowing(sh, 29)
    W = O.upcast(w)
    m = VestaGPT2(hf, batch=batch, tmax=8, per_sequence_t=True)
    x = np.array([1 if b % 3 == 1 else 2 + b for b in range(batch)], np.int32)
    ref = [O.step(sh, W, *O.new_cache(sh, 1), int(x[b]), 0)[0] for b in range(batch)]
    m.x.copy_(torch.from_numpy(x))
    m.step()
    got = m.logits().cpu().numpy()
    assert not np.isfinite(got[x == 1]).all()                    # (the rows of token 1 did overflow)
    bound = np.full(sh.N, TIGHT * (1 if batch <= 16 else 2))
    bound[1] *= 20                                               # (token 1's embedding is 20 times the others', and so is what rounding leaves of its logit)
    for b in np.flatnonzero(x != 1):
        assert (np.abs(got[b] - ref[b]) < bound).all(), b
    m.prefill(x[:, None])
    first = m.x.cpu().numpy()
    for b in np.flatnonzero(x != 1):
        if O.margin(ref[b]) > MARGIN:
            assert int(first[b]) == int(ref[b].argmax()), b


@pytest.mark.parametrize('batch', [20, 70])
def test_best_of_logits_that_are_all_minus_infinity(batch):
    """an output norm that overflows fp16 makes every logit minus infinity: all equal, so the lowest token, as the order of
    (value, lowest index) has it; tiles of 64 features (half of whose lanes hold none) and of 128"""
    from vesta_gpu_b200.gpt2 import VestaGPT2
    from vesta_gpu_b200.synth import SynthGPT2, make_weights
    sh = shape('low', L=1)
    w = make_weights(sh, 31, 'rich')
    w['wte'][:, 0] = 4                      # every state is large and positive there,
    w['lnfw'][0], w['lnfb'][0] = -10000, -65504      # the norm's output minus infinity as fp16, and so is its product with the table
    m = VestaGPT2(SynthGPT2(sh, 31, weights=w), batch=batch, tmax=8)
    m.x.copy_(torch.arange(batch, dtype=torch.int32) + 2)
    m.step()
    assert torch.isneginf(m.logits()).all()
    assert (m.next() == 0).all() and (m.x == 0).all()
    m.k.check()


def test_waits_of_a_chain_that_run_out():
    """with the limit of a wait at a nanosecond every wait that is not over within one try gives up, at different times in the
    warps of a block and in the blocks of a pair: a step of 256 rows (several tiles per block in every contraction) and prompts
    of 4,096 positions (pairs of blocks, attention on tensor memory) end with a status, publish nothing, and run again as
    before once the limit is back"""
    from vesta_gpu_b200.launch import lib, ok
    sh, batch, P = shape('wide', L=2, D=1600, H=25, F=1600, N=20000, C=64), 256, 16
    m, _ = model(sh, 41, 'rich', batch, sh.C)
    toks = np.random.RandomState(3).randint(0, sh.N, (batch, P)).astype(np.int32)
    m.prefill(toks)
    keys, vals, x = m.keys.clone(), m.vals.clone(), m.x.clone()
    m.step()
    logits, after, new = m.logits().clone(), m.x.clone(), m.keys[:, :, P].clone()
    state = dict(keys=keys, vals=vals, x=x, t=torch.tensor([P], dtype=torch.int32).cuda())
    m.load_state(state)
    nxt = m.next().clone()
    ok(lib().vesta_pass_wait_limit(m.k._pass, 1))
    m.step(2)
    assert 'operands of a contraction' in str(m.k.status())
    assert int(m.k.bar[2]) == 1 and int(m.t[0]) == P and torch.equal(m.x, x) and torch.equal(m.next(), nxt)
    ok(lib().vesta_pass_wait_limit(m.k._pass, 0))
    m.step()                                                     # (refused until the status is cleared)
    assert int(m.t[0]) == P and torch.equal(m.x, x)
    m.k.clear_status()
    m.load_state(state)
    m.step()
    m.k.check()
    assert int(m.t[0]) == P + 1 and (m.logits() - logits).abs().max() < 2 * TIGHT
    assert (m.keys[:, :, P].float() - new.float()).abs().max() <= 4e-3
    eng, = m._prefill_engines.values()
    ok(lib().vesta_pass_wait_limit(eng.h, 1))
    with pytest.raises(RuntimeError, match='gave up'):
        m.prefill(toks)
    ok(lib().vesta_pass_wait_limit(eng.h, 0))
    m.prefill(toks)
    assert int(m.t[0]) == P
    for got, ref in ((m.keys, keys), (m.vals, vals)):
        assert (got[:, :, :P].float() - ref[:, :, :P].float()).abs().max() <= 4e-3 and not got[:, :, P:].any()


def moved(t):
    """the same values two bytes behind a 16-byte boundary"""
    v = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    assert v.data_ptr() % 16 == 2
    return v.copy_(t)


@pytest.mark.parametrize('batch', [3, 12, 1, 5])
def test_weights_off_a_16_byte_boundary(batch):
    """weights that are views into a larger buffer, in the persistent kernel (one and five sequences) and in both chains: read through aligned
    copies that pack() renews; the caches are refused"""
    from vesta_gpu_b200.launch import Kernel
    sh = shape('moved')
    m, _ = model(sh, 3, 'rich', batch, 20)
    assert (m.k.few, m.k.chain) == (batch == 3, batch == 12)
    k = Kernel(m.low, device=m.device.index)
    R = dict(m.k.keep)
    for role in ('ln1w', 'ln1b', 'qkvw', 'qkvb', 'ow', 'ob', 'ln2w', 'ln2b', 'fcw', 'fcb', 'pw', 'pb', 'lnfw', 'lnfb', 'wpe'):
        R[role] = moved(R[role])
    for name in ('x', 't', 'keys', 'vals'):
        R[name] = R[name].clone()
    m.x.fill_(7)
    R['x'].fill_(7)
    k.bind(R)
    m.step()
    k.launch()
    assert (m.logits() - k.view('logit')).abs().max() < TIGHT and torch.equal(m.t, R['t'])
    for W in (m.k.keep, R):                                      # changed in place
        W['lnfw'].mul_(0.5)
        W['fcw'].mul_(2)
    m.k.pack()
    k.pack()
    m.step()
    k.launch()
    assert (m.logits() - k.view('logit')).abs().max() < TIGHT
    k.check()
    with pytest.raises(RuntimeError):
        k.bind(dict(R, keys=moved(R['keys'])))


@pytest.mark.parametrize('batch', [1, 2, 4])
def test_packing_the_matrices_of_other_tensors(batch):
    """pack(residue) makes the packed weights from the tensors that it is given, in the persistent kernel and in the chain of few
    sequences, also from views off a 16-byte boundary, until pack() or bind() makes them from the bound ones again; before the first bind
    there is nothing to keep"""
    from vesta_gpu_b200.launch import Kernel
    sh = shape('other')
    m, _ = model(sh, 3, 'rich', batch, 20)
    k = Kernel(m.low, device=m.device.index)
    R = dict(m.k.keep)
    k.pack(R)
    other = dict(R, fcw=moved(R['fcw'] * 2), qkvw=R['qkvw'] * -1)

    def logits(W):
        k.bind(dict(W, x=torch.full_like(R['x'], 7), t=torch.zeros_like(R['t']), keys=torch.zeros_like(R['keys']), vals=torch.zeros_like(R['vals'])))
        return again()

    def again():
        k.keep['t'].zero_()
        k.keep['x'].fill_(7)
        k.launch()
        k.check()
        return k.view('logit').clone()
    plain, want = logits(R), logits(dict(other, fcw=other['fcw'].clone()))
    assert (plain - want).abs().max() > 20 * TIGHT
    assert (logits(R) - plain).abs().max() < TIGHT
    k.pack(other)
    assert (again() - want).abs().max() < TIGHT
    k.pack()
    assert (again() - plain).abs().max() < TIGHT


def test_prompts_with_weights_off_a_16_byte_boundary():
    """a state dict of views (position table, output norm): prefill reads what the weights are when it is called"""
    from vesta_gpu_b200.gpt2 import VestaGPT2
    sh = shape('moved')
    m, hf = model(sh, 3, 'rich', 2, 20)

    class Views:
        def state_dict(self):
            return {n: moved(t.cuda()) if n in ('transformer.wpe.weight', 'transformer.ln_f.weight', 'transformer.ln_f.bias') else t
                    for n, t in hf.state_dict().items()}
    v = VestaGPT2(Views(), batch=2, tmax=20)
    assert v.W['wpe'].data_ptr() % 16 == 2
    toks = np.arange(24, dtype=np.int32).reshape(2, 12)
    for _ in range(2):
        m.prefill(toks)
        v.prefill(toks)
        assert (m.keys.float() - v.keys.float()).abs().max() <= 4e-3 and m.keys.any()
        for w in (m, v):
            w.W['wpe'].mul_(-1)


@pytest.mark.parametrize('batch', [12, 70])
def test_the_persistent_kernel_of_a_chain_by_its_argument_list(batch):
    """Kernel.fn and Kernel.args belong together also where steps run as a chain: launched by hand they do the same step"""
    import ctypes
    from vesta_gpu_b200.launch import lib, ok
    sh = shape('by hand')
    m, _ = model(sh, 3, 'rich', batch, 20)
    k, x = m.k, torch.arange(batch, dtype=torch.int32).cuda()
    vals, kinds = k.args
    assert k.chain and len(vals) == len(kinds) == len(m.low.params) + 7
    m.x.copy_(x)
    m.step()
    logits, after = m.logits().clone(), m.x.clone()
    m.reset()
    m.x.copy_(x)
    store = (ctypes.c_ulonglong * len(vals))(*vals)
    at = (ctypes.c_void_p * len(vals))(*[ctypes.addressof(store) + 8 * i for i in range(len(vals))])
    ok(lib().vesta_launch_cooperative(k.fn, k.grid, k.block, k.smem, torch.cuda.current_stream().cuda_stream, at))
    assert (m.logits() - logits).abs().max() < 2 * TIGHT and int(m.t[0]) == 1
    top = logits.topk(2, dim=1).values
    sure = top[:, 0] - top[:, 1] > MARGIN
    assert torch.equal(m.x[sure], after[sure])
    k.check()


def test_binding_a_chain_again():
    """other tensors, one call per step as the reference has it, then launches again: the same workspace throughout (a step that
    runs on another stream keeps its memory), the same steps as a model's"""
    from vesta_gpu_b200.launch import Kernel
    sh = shape('again')
    m, _ = model(sh, 3, 'rich', 12, 20)
    k = Kernel(m.low, device=m.device.index)
    own = lambda: dict(m.k.keep, **{n: torch.zeros_like(m.k.keep[n]) for n in ('x', 't', 'keys', 'vals')})
    R, S = own(), own()
    k.bind(R)
    work = k._work.data_ptr()
    k.launch()
    k(S)
    k(S)
    k.launch(2)
    k.bind(R)
    k.launch(3)
    assert k._work.data_ptr() == work and k.launches == 8
    m.step(4)
    assert int(R['t'][0]) == int(S['t'][0]) == int(m.t[0]) == 4
    for T in (R, S):
        assert (T['keys'].float() - m.keys.float()).abs().max() <= 4e-3 and torch.equal(T['x'], m.x)
    k.check()


def test_steps_of_a_chain_inside_a_captured_graph():
    """a caller's own CUDA graph of steps: the kernels of the chain one by one instead of the chain's graph"""
    sh = shape('captured')
    m, _ = model(sh, 3, 'rich', 12, 20)
    m.x.fill_(5)
    m.step(6)
    x, logits = m.x.clone(), m.logits().clone()
    g = torch.cuda.CUDAGraph()
    m.reset()
    m.x.fill_(5)
    with torch.cuda.graph(g):
        m.step(3)
    assert int(m.t[0]) == 0
    g.replay()
    g.replay()
    assert int(m.t[0]) == 6 and (m.logits() - logits).abs().max() < TIGHT and torch.equal(m.x, x)
    m.k.check()
