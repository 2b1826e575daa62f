"""Parity of the CUDA path with the reference interpreter (through the golden fixtures) and with
the CPU oracle, on a B200. Everything goes through the public API, i.e. through the C ABI."""
import numpy as np
import pytest
import torch

from helpers import load, fixture_inputs, teacher_tokens, close, TIGHT, MARGIN

pytestmark = pytest.mark.gpu


def model(sh, seed, init, batch, tmax, **kw):
    from vesta_gpu_b200.synth import SynthGPT2
    from vesta_gpu_b200.gpt2 import VestaGPT2
    hf = SynthGPT2(sh, seed, init)
    return VestaGPT2(hf, batch=batch, tmax=tmax, **kw), hf


def run_fixture(name, seqs=None, tune=None):
    """teacher-forced decode of the fixture's sequences as one batch; every step's token and every
    kept step's logits against the reference interpreter's"""
    g = load(name)
    sh, seed, init, prompts, gen, keep, stride = fixture_inputs(g)
    seqs = list(range(prompts.shape[0])) if seqs is None else seqs
    P = prompts.shape[1]
    steps = P + gen
    m, _ = model(sh, seed, init, len(seqs), steps, tune=tune)
    m.reset()
    feed = np.stack([teacher_tokens(g, i, P) for i in seqs])           # [B, steps]
    feed_d = torch.from_numpy(feed).cuda()
    worst, bad = 0.0, []
    for t in range(steps):
        m.x.copy_(feed_d[:, t])
        m.step()
        nxt = m.next().cpu().numpy().astype(np.int64)
        lg = m.logits()[:, ::stride].cpu().numpy() if t in keep else None
        for r, i in enumerate(seqs):
            if g[f'margins_{i}'][t] > MARGIN and nxt[r] != g[f'tokens_{i}'][t]:
                bad.append((i, t, int(nxt[r]), int(g[f'tokens_{i}'][t])))
            if lg is not None:
                ref = g[f'logits_{i}'][keep.index(t)]
                assert close(lg[r], ref), (name, i, t)
                worst = max(worst, float(np.abs(lg[r] - ref).max()))
    m.k.check()
    assert not bad, bad[:5]
    assert worst < TIGHT, worst
    assert int(m.t.cpu()[0]) == steps
    return worst


def test_tiny_fixture():
    run_fixture('tiny_b3')


def test_tiny3_fixture_vocab_not_multiple_of_16():
    run_fixture('tiny3_b2')


def test_gpt2_small_rich_init():
    run_fixture('gpt2_rich_b1')


@pytest.mark.parametrize('name', ['tiny_b3', 'gpt2_rich_b1'])
def test_fixed_point_sums_against_the_reference(name):
    """tune={'ordered': True}: the state vectors as 64-bit fixed point, combined with integer atomics"""
    run_fixture(name, tune=dict(ordered=True))


@pytest.mark.parametrize('batch', [1, 8])
def test_ordered_mode_gives_the_same_bits_on_every_run(batch):
    """GPT-2 small: 16 prompt tokens and 64 free-running steps, twice from the same state. With fixed-point sums (integer
    atomics: associative, so the arrival order of the partial sums does not matter) tokens, logits and the K/V cache of
    the two runs are bit-identical; the reference reduces in a fixed order (vesta/lower.py:1045-1047) for the same end."""
    from vesta_gpu_b200.shapes import GPT2_SMALL
    from vesta_gpu_b200.synth import make_prompts
    P, G = 16, 64
    prompts = torch.from_numpy(make_prompts(GPT2_SMALL, batch, P, seed=7).copy()).cuda()
    m, _ = model(GPT2_SMALL, 0, 'baseline', batch, P + G + 1, tune=dict(ordered=True))
    assert m.low.dims['ordered']

    def run():
        m.reset()
        for t in range(P):
            m.x.copy_(prompts[:, t]); m.step()
        toks = [m.x.clone()]
        for _ in range(G):
            m.step(); toks.append(m.x.clone())
        m.k.check()
        return torch.stack(toks, 1).clone(), m.logits().clone(), m.keys.clone(), m.vals.clone()
    a, b = run(), run()
    for x, y in zip(a, b):
        assert torch.equal(x, y)


def test_gpt2_small_batch1_config():
    """128-token prompt + 256 greedy steps, batch 1"""
    run_fixture('gpt2_cfg2', seqs=[0])


def test_gpt2_small_batch8_config():
    """eight sequences, 128 + 256 positions"""
    run_fixture('gpt2_cfg2')


def test_gpt2_xl_shape():
    run_fixture('gpt2_xl_b1')


@pytest.mark.parametrize('name,tune', [(n, None) for n in ('gpt2_cfg3_sample', 'gpt2_cfg5_sample', 'gpt2_xl16_sample', 'gpt2_cfg5_b64_sample', 'gpt2_cfg5_b256_sample',
                                                          'gpt2_cfg3_tail_sample', 'gpt2_xl1_sample')]
                         + [(n, dict(ln_dist=True)) for n in ('gpt2_cfg3_sample', 'gpt2_cfg5_b64_sample', 'gpt2_cfg3_tail_sample')])
def test_deep_context_samples_against_the_reference(name, tune):
    """the large-batch paths at full model size against the reference interpreter, as a chain of kernels and, where `tune` names
    the option that the persistent kernel takes by itself there, in that kernel: (cfg3) 64 sequences with 600
    positions in every cache (the persistent kernel: distributed LayerNorm, fold-slice MLP projection, several attention items
    of five tiles per CTA, tcgen05 contractions); (cfg5) ragged batches of 32, 64 and 256 (what the batch-sharded benchmark runs per
    GPU on 8, 4 and 1 GPUs) with 64..512 positions per sequence and per-sequence positions; (cfg3 tail) 64 sequences at
    positions 1021..1023 of a 1024-row cache: the last K/V tile and the last position the cache holds; (xl16, xl1) the XL
    shape at batch 16 and batch 1, context 300. Caches are seeded (synth.make_cache); the sampled sequences are compared over two
    teacher-forced steps."""
    from vesta_gpu_b200.shapes import SHAPES
    from vesta_gpu_b200.synth import make_cache
    g = load(name)
    sh, steps, stride, B = SHAPES[str(g['shape'])], int(g['steps']), int(g['stride']), int(g['batch'])
    ctxs = g['ctxs'].astype(np.int32)
    ragged = int(ctxs.min()) != int(ctxs.max())
    m, _ = model(sh, int(g['seed']), str(g['init']), B, int(ctxs.max()) + steps, per_sequence_t=ragged, tune=tune)
    assert m.k.chain == (B > 8 and not tune)
    if not m.k.chain and B >= 64:
        assert m.low.dims['tc'] and m.low.dims['ksplit'] and m.low.dims['tcl']
    m.reset()
    for b in range(B):
        k0, v0 = make_cache(sh, int(g['cache_seed_base']) + b, int(ctxs[b]))
        m.keys[b, :, :ctxs[b]].copy_(torch.from_numpy(k0)); m.vals[b, :, :ctxs[b]].copy_(torch.from_numpy(v0))
    m.t.copy_(torch.from_numpy(ctxs[:m.t.numel()])); m.x.copy_(torch.from_numpy(g['x0']))
    worst = 0.0
    for s_ in range(steps):
        if s_:
            x = m.x.cpu().numpy().copy()
            for i, b in enumerate(g['sample']):
                x[b] = g[f'fed_{i}'][s_]                          # teacher forcing for the compared sequences
            m.x.copy_(torch.from_numpy(x))
        m.step()
        lg, nx = m.logits().cpu().numpy(), m.next().cpu().numpy()
        for i, b in enumerate(g['sample']):
            ref = g[f'logits_{i}'][s_]
            assert close(lg[b][::stride], ref), (s_, b)
            worst = max(worst, float(np.abs(lg[b][::stride] - ref).max()))
            assert np.abs(lg[b][g[f'top_idx_{i}'][s_]] - g[f'top_val_{i}'][s_]).max() < 5e-3
            if g[f'margins_{i}'][s_] > MARGIN:
                assert int(nx[b]) == int(g[f'tokens_{i}'][s_]), (s_, b)
    m.k.check()
    print(f'{name}: max |logit - reference| = {worst:.2e}')
    assert worst < 5e-3, worst          # fp16-head operands at these batches: a few 1e-3, far inside the 2e-2 rule


def test_free_running_feedback_matches_reference_tokens():
    """feedback on, no host write between generated steps: the stream equals the reference's up to the
    first step whose margin is below the bar"""
    g = load('gpt2_cfg2')
    sh, seed, init, prompts, gen, keep, stride = fixture_inputs(g)
    B, P = prompts.shape
    m, _ = model(sh, seed, init, B, P + gen)
    m.reset()
    pd = torch.from_numpy(prompts).cuda()
    for t in range(P):
        m.x.copy_(pd[:, t]); m.step()
    toks = [m.x.clone()]
    for _ in range(gen - 1):
        m.step(); toks.append(m.x.clone())
    got = torch.stack(toks, 1).cpu().numpy()
    m.k.check()
    for i in range(B):
        ref = g[f'tokens_{i}'][P - 1:P - 1 + gen]
        sure = g[f'margins_{i}'][P - 1:P - 1 + gen] > MARGIN
        stop = gen if sure.all() else int(np.argmin(sure))
        assert np.array_equal(got[i, :stop + 0], ref[:stop]), i


@pytest.mark.parametrize('batch', [1, 2, 5, 8])
def test_against_oracle_other_batches(batch):
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY3
    from vesta_gpu_b200.synth import make_prompts
    steps = 9
    m, hf = model(TINY3, 11, 'rich', batch, steps)
    W = O.upcast(hf.weights)
    feed = make_prompts(TINY3, batch, steps, seed=batch)
    caches = [O.new_cache(TINY3, steps) for _ in range(batch)]
    m.reset()
    for t in range(steps):
        m.x.copy_(torch.from_numpy(feed[:, t].copy()).cuda()); m.step()
        lg = m.logits().cpu().numpy(); nx = m.next().cpu().numpy()
        for i in range(batch):
            ref, rn = O.step(TINY3, W, caches[i][0], caches[i][1], int(feed[i, t]), t)
            assert np.abs(lg[i] - ref).max() < TIGHT
            if O.margin(ref) > MARGIN:
                assert int(nx[i]) == rn
    # the cache holds the fp16-rounded K and V of every position (gpt2.vst:48-49); allow one fp16 step
    k = m.keys.cpu().numpy().astype(np.float32)
    for i in range(batch):
        ref = caches[i][0].astype(np.float32)
        assert np.abs(k[i, :, :steps] - ref).max() <= 2e-3
    m.k.check()


@pytest.mark.parametrize('batch,ctx,tune', [(8, 3, None), (8, 40, None), (7, 40, dict(fuse_proj=False, nch=2)), (8, 40, dict(ordered=True)), (2, 40, None)])
def test_more_attention_items_than_ctas_at_small_batch(batch, ctx, tune):
    """twenty heads: 160 (sequence, head) pairs at eight sequences, so twelve CTAs hold two attention items per layer (and,
    in the fused mode, apply the projection of two heads); short and longer contexts, the unfused mode with two position
    chunks per pair, fixed-point sums; against the oracle on seeded caches"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import HEADS20 as sh
    from vesta_gpu_b200.synth import make_cache
    steps = 3
    m, hf = model(sh, 17, 'rich', batch, ctx + steps, tune=tune)
    assert m.low.dims['kernel'] == 'small'
    W = O.upcast(hf.weights)
    caches = []
    m.reset()
    for b in range(batch):
        k0, v0 = make_cache(sh, 500 + b, ctx)
        ck, cv = O.new_cache(sh, ctx + steps)
        ck[:, :ctx] = k0; cv[:, :ctx] = v0
        caches.append((ck, cv))
        m.keys[b, :, :ctx].copy_(torch.from_numpy(k0)); m.vals[b, :, :ctx].copy_(torch.from_numpy(v0))
    m.t.fill_(ctx)
    x = np.array([(b * 37 + 5) % sh.N for b in range(batch)], np.int32)
    for s_ in range(steps):
        m.x.copy_(torch.from_numpy(x)); m.step()
        lg, nx = m.logits().cpu().numpy(), m.next().cpu().numpy()
        for b in range(batch):
            ref, rn = O.step(sh, W, caches[b][0], caches[b][1], int(x[b]), ctx + s_)
            assert np.abs(lg[b] - ref).max() < TIGHT, (s_, b)
            if O.margin(ref) > MARGIN:
                assert int(nx[b]) == rn
            x[b] = rn
    m.k.check()


@pytest.mark.parametrize('batch,slab_tiles,tune', [
    (20, 1, None), (20, None, None), (9, 1, None), (33, 2, None),
    (20, 1, dict(ln_dist=True, act_lo=True)),          # rows normalised once on the grid, tiles through global memory
    (33, 2, dict(ln_dist=True, act_lo=False)),         # ... with fp16-head operand tiles (the large-batch mode)
    (5, None, dict(ln_dist=True)),                     # ... at a batch below one tile
    (20, 1, dict(ln_dist=False, act_lo=True)),         # every CTA normalises its slab, head + remainder
    (60, None, None),                                  # more (sequence, head) items than CTAs: several per CTA
    (60, None, dict(tail_split=4)),                    # ... the items of the last round split into four position chunks
    (60, None, dict(kv_stages=2, nch=2)),              # ... with two K/V stages and two position chunks per item
    (64, None, dict(tc=True)),                         # 64 sequences and more: logits on tcgen05 / tensor memory
    (70, None, dict(tc=True)),                                # ... two slabs of 64 sequences, the second ragged
    (70, None, dict(tc=False)),                        # ... and the same batch on the mma.sync path
    (33, 2, dict(ksplit=False)),                       # large batch with the projections as wide fold slices (148-way sums)
    (9, 1, dict(ksplit=True)),                         # small batch with the projections as deep fold slices, GELU through global memory
    (20, None, dict(ksplit=True, ln_dist=False)),      # ... with every CTA normalising its own rows
])
def test_batches_above_one_slab(batch, slab_tiles, tune):
    """batches larger than the operand tiles in shared memory run slab by slab (the last slab ragged), in both
    LayerNorm modes and both operand precisions"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY3
    from vesta_gpu_b200.synth import make_prompts
    steps = 5
    m, hf = model(TINY3, 11, 'rich', batch, steps, slab_tiles=slab_tiles, tune=tune)
    W = O.upcast(hf.weights)
    feed = make_prompts(TINY3, batch, steps, seed=batch)
    caches = [O.new_cache(TINY3, steps) for _ in range(batch)]
    m.reset()
    for t in range(steps):
        m.x.copy_(torch.from_numpy(feed[:, t].copy()).cuda()); m.step()
        lg = m.logits().cpu().numpy(); nx = m.next().cpu().numpy()
        for i in range(batch):
            ref, rn = O.step(TINY3, W, caches[i][0], caches[i][1], int(feed[i, t]), t)
            assert np.abs(lg[i] - ref).max() < TIGHT, (t, i)
            if O.margin(ref) > MARGIN:
                assert int(nx[i]) == rn
    m.k.check()


@pytest.mark.parametrize('batch,tune', [
    (64, None),                                         # one slab of 64 sequences
    (70, None),                                         # two slabs, the second with six live rows
    (130, None),                                        # three row blocks of 64, the last with two live rows
    (64, dict(tcl_rb=32)),                              # two row blocks of 32
    (130, dict(tcl_rb=32, tcl_nw=16)),                  # five row blocks of 32 x units of 16 output columns
    (64, dict(tcl_rb=64, tcl_nw=16)),                   # one row block: every CTA reads the operand of all 64 sequences
    (64, dict(tc_layers=False)),                        # the same batch with the layer contractions on mma.sync
])
def test_tensor_core_layer_contractions(batch, tune):
    """64 sequences and more: QKV, attention projection, FC and MLP projection as tcgen05 units (a block of sequences as
    the rows of the product, accumulators in tensor memory, weights from the packed operand image, operands written by
    the previous phase as fp16 swizzled rows), against the oracle over several steps (K/V emit and attention included)"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY
    from vesta_gpu_b200.synth import make_prompts
    steps = 6
    m, hf = model(TINY, 11, 'rich', batch, steps, tune=dict(tune or {}, ln_dist=True))     # (rows normalised once on the grid, as at full size)
    assert bool(m.low.dims['tcl']) == (not tune or tune.get('tc_layers', True))
    W = O.upcast(hf.weights)
    feed = make_prompts(TINY, batch, steps, seed=batch)
    caches = [O.new_cache(TINY, steps) for _ in range(batch)]
    m.reset()
    worst = 0.0
    for t in range(steps):
        m.x.copy_(torch.from_numpy(feed[:, t].copy()).cuda()); m.step()
        lg = m.logits().cpu().numpy(); nx = m.next().cpu().numpy()
        for i in range(batch):
            ref, rn = O.step(TINY, W, caches[i][0], caches[i][1], int(feed[i, t]), t)
            worst = max(worst, float(np.abs(lg[i] - ref).max()))
            if O.margin(ref) > MARGIN:
                assert int(nx[i]) == rn, (t, i)
    assert worst < TIGHT, worst
    k = m.keys.cpu().numpy().astype(np.float32)
    for i in range(batch):
        assert np.abs(k[i, :, :steps] - caches[i][0].astype(np.float32)).max() <= 2e-3
    m.k.check()


@pytest.mark.parametrize('B', [6, 12])
def test_ragged_prompts_fed_on_the_device(B):
    """in the persistent kernel and in a chain: per-sequence prompt lengths, consumed by the kernel's own feedback (no host write between steps),
    late starts so that every prompt ends at the same step; the greedy streams equal the oracle's"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY3
    from vesta_gpu_b200.synth import make_ragged_prompts
    gen = 8
    lens, toks = make_ragged_prompts(TINY3, B, 1, 9, seed=3)
    pmax = int(lens.max()); steps = pmax + gen
    m, hf = model(TINY3, 11, 'rich', B, steps, per_sequence_t=True, prompt_len=pmax)
    W = O.upcast(hf.weights)
    m.reset()
    m.prompt.copy_(torch.from_numpy(toks[:, :pmax].copy())); m.plen.copy_(torch.from_numpy(lens))
    start = (lens - pmax).astype(np.int32)
    m.t.copy_(torch.from_numpy(start)); m.x.copy_(torch.from_numpy(np.where(start == 0, toks[:, 0], 0).astype(np.int32)))
    got = []
    for _ in range(steps - 1):
        m.step(); got.append(m.x.clone())
    got = torch.stack(got, 1).cpu().numpy()
    m.k.check()
    assert m.t.cpu().numpy().tolist() == (lens + gen - 1).tolist()
    for i in range(B):
        r = O.decode(TINY3, W, toks[i, :lens[i]], gen)
        mine = got[i, pmax - 1: pmax - 1 + gen - 1]
        ref = r['tokens'][lens[i] - 1: lens[i] - 1 + gen - 1]
        sure = r['margins'][lens[i] - 1: lens[i] - 1 + gen - 1] > MARGIN
        stop = len(ref) if sure.all() else int(np.argmin(sure))
        assert np.array_equal(mine[:stop], ref[:stop]), i


@pytest.mark.parametrize('B', [4, 6])                    # (the chain of few sequences, the persistent kernel)
def test_per_sequence_positions_ragged_starts(B):
    """every sequence at its own position: sequence b starts b*2 steps late"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY
    from vesta_gpu_b200.synth import make_prompts
    steps = 12
    m, hf = model(TINY, 3, 'rich', B, steps, per_sequence_t=True, feedback=False)
    assert m.k.graphs == (B == 4)
    W = O.upcast(hf.weights)
    feed = make_prompts(TINY, B, steps, seed=9)
    caches = [O.new_cache(TINY, steps) for _ in range(B)]
    m.reset()
    for s in range(steps):
        pos = np.array([max(0, s - 2 * b) for b in range(B)], np.int32)
        live = [s >= 2 * b for b in range(B)]
        x = np.array([feed[b, pos[b]] for b in range(B)], np.int32)
        m.x.copy_(torch.from_numpy(x).cuda()); m.t.copy_(torch.from_numpy(pos).cuda())
        m.step()
        lg = m.logits().cpu().numpy()
        for b in range(B):
            if live[b]:
                ref, _ = O.step(TINY, W, caches[b][0], caches[b][1], int(x[b]), int(pos[b]))
                assert np.abs(lg[b] - ref).max() < TIGHT, (s, b)
    m.k.check()


def test_batch_rows_are_independent_at_full_size():
    """the same prompt in all 8 rows gives the same tokens in every row, equal to the batch-1 run"""
    from vesta_gpu_b200.shapes import GPT2_SMALL
    from vesta_gpu_b200.synth import make_prompts
    P, G = 16, 24
    prompt = make_prompts(GPT2_SMALL, 1, P, seed=5)[0]
    outs = {}
    for B in (1, 8):
        m, _ = model(GPT2_SMALL, 0, 'baseline', B, P + G)
        m.reset()
        for t in range(P):
            m.x.fill_(int(prompt[t])); m.step()
        first = m.logits().clone()
        toks = [m.x.clone()]
        for _ in range(G - 1):
            m.step(); toks.append(m.x.clone())
        outs[B] = (torch.stack(toks, 1).cpu().numpy(), first.cpu().numpy())
        m.k.check()
        del m
    t8, l8 = outs[8]
    assert all(np.array_equal(t8[0], t8[r]) for r in range(8))
    assert np.abs(l8 - l8[0:1]).max() < 1e-4
    assert np.abs(l8[0] - outs[1][1][0]).max() < 1e-4
    assert np.array_equal(t8[0], outs[1][0][0])


def test_tensor_core_logits_at_full_size_equal_the_mma_path():
    """GPT-2 small, 64 sequences, one step on a filled cache: the tcgen05 logits (128 x 64 tiles of the whole
    vocabulary, every CTA's range ragged at its end) against the mma.sync path on the same inputs, and the
    arg-max of each sequence against its own logits"""
    from vesta_gpu_b200.shapes import GPT2_SMALL
    B, ctx = 64, 40
    outs = []
    for tc in (True, False):
        m, _ = model(GPT2_SMALL, 0, 'rich', B, ctx + 2, tune=dict(tc=tc))
        assert bool(m.low.dims['tc']) == tc
        m.reset()
        g = torch.Generator(device='cuda').manual_seed(3)
        m.keys[:, :, :ctx].copy_((torch.randn(m.keys[:, :, :ctx].shape, generator=g, device='cuda') * 0.3).half())
        m.vals[:, :, :ctx].copy_((torch.randn(m.vals[:, :, :ctx].shape, generator=g, device='cuda') * 0.3).half())
        m.t.fill_(ctx); m.x.copy_(torch.arange(B, dtype=torch.int32, device='cuda') * 97 + 11)
        m.step(); m.k.check()
        lg, nx = m.logits().cpu().numpy().copy(), m.next().cpu().numpy().copy()
        assert np.array_equal(nx.astype(np.int64), lg.argmax(1))
        outs.append(lg)
        del m
    # both paths round the activations to fp16 (each within ~1e-3 of the fp32-activation result over 3.2 M logits)
    assert np.abs(outs[0] - outs[1]).max() < 5e-3


@pytest.mark.parametrize('batch', [3, 5])                # (the chain of few sequences, the persistent kernel)
def test_multi_step_launch_and_reset(batch):
    from vesta_gpu_b200.shapes import TINY
    m, _ = model(TINY, 3, 'rich', batch, 32)
    assert m.k.graphs == (batch == 3)
    def run(chunked):
        m.reset(); m.x.copy_(torch.arange(1, batch + 1, dtype=torch.int32))
        if chunked:
            m.step(20)
        else:
            for _ in range(20):
                m.step()
        return m.x.cpu().numpy().copy(), m.logits().cpu().numpy().copy(), int(m.t.cpu()[0])
    a, b = run(False), run(True)
    assert np.array_equal(a[0], b[0]) and a[2] == b[2] == 20
    assert np.abs(a[1] - b[1]).max() < 1e-4
    m.k.check()


@pytest.mark.parametrize('per_launch', [1, 3, 7, 20])
def test_steps_inside_one_launch_equal_separate_launches(per_launch):
    """several decode steps inside one launch (the kernel feeds itself and waits on its step flag) against
    one launch per step: same tokens, same positions, same cache; ragged prompts fed on the device included"""
    from vesta_gpu_b200.shapes import TINY3
    from vesta_gpu_b200.synth import make_ragged_prompts
    B, steps = 5, 20
    lens, toks = make_ragged_prompts(TINY3, B, 1, 6, seed=5)
    pmax = int(lens.max())
    m, _ = model(TINY3, 7, 'rich', B, steps + 1, per_sequence_t=True, prompt_len=pmax)
    def run(per):
        m.reset(); m.k.bar.zero_()
        m.prompt.copy_(torch.from_numpy(toks[:, :pmax].copy())); m.plen.copy_(torch.from_numpy(lens))
        start = (lens - pmax).astype(np.int32)
        m.t.copy_(torch.from_numpy(start)); m.x.copy_(torch.from_numpy(np.where(start == 0, toks[:, 0], 0).astype(np.int32)))
        m.k.launch(steps, per_launch=per)
        m.k.check()
        return m.x.cpu().numpy().copy(), m.t.cpu().numpy().copy(), m.logits().cpu().numpy().copy(), m.keys.float().cpu().numpy().copy()
    a, b = run(1), run(per_launch)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert np.abs(a[2] - b[2]).max() < 2e-3 and np.abs(a[3] - b[3]).max() < 2e-3
    assert int(m.k.bar[3]) == 0 and int(m.k.bar[32]) == 0           # step flag and barrier counter left clear


@pytest.mark.parametrize('batch', [2, 5])                # (the chain of few sequences, the persistent kernel)
def test_launch_of_many_steps_stops_at_the_end_of_the_cache(batch):
    """a launch asked for more steps than the cache has room for stops after the last step that fits and
    says so; the steps before it are complete and the kernel is usable again afterwards"""
    from vesta_gpu_b200.shapes import TINY
    m, _ = model(TINY, 3, 'rich', batch, 8)
    assert m.k.graphs == (batch == 2)
    m.reset(); m.x.fill_(3)
    m.k.launch(7, per_launch=1)
    want_x, want_logits = m.x.clone(), m.logits().clone()
    m.k.launch(1)                                   # the 8th step fills the cache: t becomes 8
    full_x = m.x.clone()
    m.reset(); m.x.fill_(3)
    m.k.launch(20, per_launch=20)
    assert 'out of range' in str(m.k.status())
    assert int(m.t.cpu()[0]) == 8 and torch.equal(m.x, full_x)
    m.k.bar.zero_(); m.reset(); m.x.fill_(3)
    m.k.launch(7, per_launch=7)
    m.k.check()
    assert torch.equal(m.x, want_x) and (m.logits() - want_logits).abs().max() < 2e-3


@pytest.mark.parametrize('batch', [4, 6])                # (the chain of few sequences, the persistent kernel)
def test_host_driven_step_equals_the_device_loop(batch):
    """vesta_step_host (tokens from pinned host memory, chosen tokens back to it, one call per step) against the
    kernel feeding itself"""
    from vesta_gpu_b200.shapes import TINY3
    m, _ = model(TINY3, 5, 'rich', batch, 12)
    assert m.k.graphs == (batch == 4)
    start = torch.tensor([3, 50, 200, 331, 17, 90][:batch], dtype=torch.int32)
    m.reset(); m.x.copy_(start); m.k.launch(10, per_launch=1)
    want_x, want_logits = m.x.cpu(), m.logits().cpu()
    hx, hn = start.clone().pin_memory(), torch.empty(batch, dtype=torch.float32).pin_memory()
    m.reset()
    for _ in range(10):
        m.step_host(hx, hn)
        hx.copy_(hn.to(torch.int32))
    m.k.check()
    assert torch.equal(hx, want_x) and torch.equal(m.x.cpu(), want_x)
    assert (m.logits().cpu() - want_logits).abs().max() < 2e-3


def test_prefill_in_one_call_and_state_round_trip():
    """prefill_stepwise() (prompts to the device once, the kernel feeds itself) against feeding the prompt token by token from
    the host; state() / load_state() carry a generation over to a second model"""
    from vesta_gpu_b200.shapes import TINY3
    from vesta_gpu_b200.synth import make_ragged_prompts
    B, gen = 4, 6
    lens, toks = make_ragged_prompts(TINY3, B, 2, 7, seed=9)
    pmax = int(lens.max())
    m, hf = model(TINY3, 13, 'rich', B, pmax + gen + 1, per_sequence_t=True, prompt_len=pmax)
    m.prefill_stepwise(toks[:, :pmax], lens)
    m.k.check()
    first = m.x.cpu().numpy().copy()
    assert m.t.cpu().numpy().tolist() == lens.tolist()
    # the same prompts, one sequence at a time, token by token
    m1, _ = model(TINY3, 13, 'rich', 1, pmax + gen + 1)
    for i in range(B):
        m1.reset()
        for p in range(int(lens[i])):
            m1.x.fill_(int(toks[i, p])); m1.step()
        assert int(m1.x.cpu()[0]) == int(first[i]), i
    # carry on, save in the middle, finish on a second model
    m.step(2)
    st = m.state()
    m.step(gen - 2)
    want = m.x.cpu().numpy().copy()
    m2, _ = model(TINY3, 13, 'rich', B, pmax + gen + 1, per_sequence_t=True, prompt_len=pmax)
    m2.prompt.copy_(m.prompt); m2.plen.copy_(m.plen)
    m2.load_state(st)
    m2.step(gen - 2)
    m2.k.check()
    assert np.array_equal(m2.x.cpu().numpy(), want)
    with pytest.raises(ValueError):
        m2.load_state(dict(st, x=st['x'][:2]))


@pytest.mark.parametrize('shape_name,batch,rows', [('tiny', 5, 128), ('tiny3', 3, 64), ('tiny', 9, 64)])
def test_dense_prefill_equals_the_oracle(shape_name, batch, rows):
    """prefill(): every prompt position of every sequence as a row of a dense pass (rows of one sequence attend to the
    rows before them, written in the same launch; several launches when the prompts exceed `rows`). Cache, first
    generated token and the tokens that follow against the oracle, ragged lengths included."""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import SHAPES
    from vesta_gpu_b200.synth import make_ragged_prompts
    sh = SHAPES[shape_name]
    gen = 4
    lens, toks = make_ragged_prompts(sh, batch, 3, 40, seed=batch)
    pmax = int(lens.max())
    m, hf = model(sh, 21, 'rich', batch, pmax + gen + 1, per_sequence_t=True)
    m.prefill(toks[:, :pmax], lens, rows=rows)
    m.k.check()
    assert m.t.cpu().numpy().tolist() == lens.tolist()
    assert list(m._prefill_engines) == [rows]                         # one pass object of so many rows read them all
    W = O.upcast(hf.weights)
    first = m.x.cpu().numpy()
    keys = m.keys.float().cpu().numpy()
    got = [m.x.clone()]
    for _ in range(gen - 1):
        m.step(); got.append(m.x.clone())
    got = torch.stack(got, 1).cpu().numpy()
    for i in range(batch):
        r = O.decode(sh, W, toks[i, :lens[i]], gen)
        k_ref = np.zeros_like(keys[i])
        # the oracle's cache of the prompt positions (decode() keeps it internally: rebuild it step by step)
        ck, cv = O.new_cache(sh, int(lens[i]))
        for p in range(int(lens[i])):
            O.step(sh, W, ck, cv, int(toks[i, p]), p)
        assert np.abs(keys[i, :, :lens[i]] - ck.astype(np.float32)).max() <= 4e-3, i
        ref = r['tokens'][lens[i] - 1: lens[i] - 1 + gen]
        sure = r['margins'][lens[i] - 1: lens[i] - 1 + gen] > MARGIN
        stop = len(ref) if sure.all() else int(np.argmin(sure))
        assert np.array_equal(got[i, :stop], ref[:stop]), (i, got[i], ref)


@pytest.mark.parametrize('rows', [None, 256])
def test_dense_prefill_at_full_size_against_the_reference(rows):
    """GPT-2 small, the eight 128-token prompts of the batch-8 fixture in one dense pass (one launch of 1024 rows by
    default, or 4 launches of 256; tensor-core contractions; logits only for the slab that holds the last positions): the
    first generated token of every sequence and the free-running tokens after it equal the reference interpreter's
    wherever its margin is above the bar"""
    g = load('gpt2_cfg2')
    sh, seed, init, prompts, gen, keep, stride = fixture_inputs(g)
    B, P = prompts.shape
    m, _ = model(sh, seed, init, B, P + 16)
    m.prefill(prompts, rows=rows)
    eng, = m._prefill_engines.values()
    assert eng.R == (rows or 1024)
    from vesta_gpu_b200.passes import tiles
    full = [t[0] for k, t in tiles(eng.desc, eng.R, B).items() if k != 'logits']
    assert rows or min(full) >= 128, full                             # 1,024 rows: products of 128 features and more in every layer contraction
    toks = [m.x.clone()]
    for _ in range(11):
        m.step(); toks.append(m.x.clone())
    got = torch.stack(toks, 1).cpu().numpy()
    m.k.check()
    compared = 0
    for i in range(B):
        ref = g[f'tokens_{i}'][P - 1:P - 1 + 12]
        sure = g[f'margins_{i}'][P - 1:P - 1 + 12] > MARGIN
        stop = 12 if sure.all() else int(np.argmin(sure))
        assert np.array_equal(got[i, :stop], ref[:stop]), (i, got[i], ref)
        compared += stop
    assert compared >= 4 * B


@pytest.mark.parametrize('batch,tune', [(3, None), (70, dict(ln_dist=True)), (70, None), (12, None), (5, None)])
@pytest.mark.parametrize('without', [('qkvb', 'fcb'), ('ln1b', 'qkvb', 'ob', 'ln2b', 'fcb', 'pb', 'lnfb')])
def test_program_without_shifts_or_biases(batch, tune, without):
    """a program that leaves out additive parameters (both kernel texts, at 70 sequences the tensor-core contractions, and both
    chains) and the same tokens as prompts: the kernel reads zeros in their place; against the oracle with those parameters set
    to zero, which is the same arithmetic as the shorter statements"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY
    from vesta_gpu_b200.synth import make_prompts
    steps = 5
    m, hf = model(TINY, 5, 'rich', batch, steps, without=without, tune=tune)
    assert m.k.chain == (batch > 8 and not tune) and m.k.few == (batch == 3)
    assert m.low.dims['absent'] == sorted(without) and not set(without) & set(m.W)
    weights = dict(hf.weights)
    for n in without:
        weights[n] = np.zeros_like(weights[n])
    W = O.upcast(weights)
    feed = make_prompts(TINY, batch, steps, seed=batch)
    caches = [O.new_cache(TINY, steps) for _ in range(batch)]
    m.reset()
    for t in range(steps):
        m.x.copy_(torch.from_numpy(feed[:, t].copy()).cuda()); m.step()
        lg = m.logits().cpu().numpy(); nx = m.next().cpu().numpy()
        for i in range(0, batch, max(1, batch // 6)):
            ref, rn = O.step(TINY, W, caches[i][0], caches[i][1], int(feed[i, t]), t)
            assert np.abs(lg[i] - ref).max() < TIGHT, (t, i)
            if O.margin(ref) > MARGIN:
                assert int(nx[i]) == rn
    keys, vals = m.keys.float(), m.vals.float()
    m.prefill(feed)
    assert (m.keys.float() - keys).abs().max() <= 4e-3 and (m.vals.float() - vals).abs().max() <= 4e-3
    m.k.check()


@pytest.mark.parametrize('batch', [2, 5])                # (the chain of few sequences, the persistent kernel)
def test_out_of_range_inputs_are_refused_not_executed(batch):
    from vesta_gpu_b200.shapes import TINY
    m, _ = model(TINY, 3, 'rich', batch, 8)
    assert m.k.graphs == (batch == 2)
    m.reset(); m.x.fill_(3); m.step()
    before = m.logits().clone()
    m.t.fill_(8)                                  # position == tmax: outside the cache
    m.step()
    assert 'out of range' in str(m.k.status())
    assert torch.equal(before, m.logits())        # nothing ran
    with pytest.raises(RuntimeError):
        m.k.check()
    m.k.clear_status(); m.t.fill_(1); m.x.fill_(TINY.N)      # token id == vocabulary size
    m.step()
    assert 'out of range' in str(m.k.status())
    m.k.clear_status(); m.x.fill_(3); m.step()
    assert m.k.status() == 0


@pytest.mark.parametrize('batch', [2, 20])
def test_a_wait_that_runs_out_ends_the_launch_with_a_status(batch):
    """Every wait in the kernels is bounded. Here the grid barrier's counter is preset so that the first barrier can
    never be satisfied and the limit is lowered to 2 ms: the launch must return, say where it gave up, leave its
    counters clear, refuse further launches until the host clears the status, and then work again. (Both kernel
    texts: at most eight sequences, and more.)"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.shapes import TINY3
    m, hf = model(TINY3, 11, 'rich', batch, 6, tune=dict(wait_ns=2_000_000))
    m.reset(); m.x.fill_(3)
    m.k.bar[32] = -(2 ** 31)                       # the counter all CTAs poll: never reaches generation x CTAs
    m.step()
    torch.cuda.synchronize()                        # returns: nothing hangs
    # the consumers' barrier wait and the producer thread's wait for them run out at about the same time: either may report
    assert any(w in str(m.k.status()) for w in ('grid barrier', 'producer')), m.k.status()
    bar = m.k.bar.cpu().numpy()
    assert bar[2] == 1 and bar[1] == 0 and bar[3] == 0 and bar[32] == 0     # abort raised; arrivals, step flag and barrier counter left clear
    with pytest.raises(RuntimeError):
        m.k.check()
    # sticky: the next launch does nothing at all
    m.reset(); m.x.fill_(3)
    m.step(); torch.cuda.synchronize()
    assert int(m.t.cpu()[0]) == 0 and int(m.x.cpu()[0]) == 3
    # cleared: a normal step, equal to the oracle's
    m.k.clear_status()
    m.step(); m.k.check()
    W = O.upcast(hf.weights)
    k0, v0 = O.new_cache(TINY3, 6)
    ref, rn = O.step(TINY3, W, k0, v0, 3, 0)
    assert np.abs(m.logits().cpu().numpy()[0] - ref).max() < TIGHT and int(m.t.cpu()[0]) == 1


def test_kernel_api_mirrors_reference():
    """vesta/launch.py:29-73: attributes, view(), bind() assertions"""
    from vesta_gpu_b200.shapes import TINY
    from vesta_gpu_b200.launch import Kernel
    m, _ = model(TINY, 3, 'rich', 2, 8)
    k = m.k
    for attr in ('mod', 'fn', 'smem', 'sms', 'grid', 'block', 'lowered', 'S', 'bar', 'TS', 'args', 'keep'):
        assert hasattr(k, attr), attr
    assert k.grid == k.sms == torch.cuda.get_device_properties(0).multi_processor_count
    k2 = Kernel(m.low, block=256, device=0)               # the reference's default block size is accepted and means the lowered one
    assert k2.block == m.low.block
    with pytest.warns(RuntimeWarning):
        Kernel(m.low, blocks_per_sm=4)
    with pytest.raises(RuntimeError):
        Kernel(m.low, block=128)
    assert k.view('logit').shape == (2, TINY.N) and k.view('next').shape == (2,)
    assert k.view('next').dtype == torch.float32
    R = dict(k.keep)
    R['wte'] = R['wte'].t().contiguous().t()      # same values, not contiguous
    with pytest.raises(AssertionError):
        k.bind(R)
    R['wte'] = k.keep['wte'].float()
    with pytest.raises(AssertionError):
        k.bind(R)
    assert m.weight_bytes == TINY.weight_bytes() and m.kv_bytes(5) == 2 * TINY.L * 2 * 5 * TINY.D * 2


def test_rows_of_prompts_in_the_persistent_kernel():
    """lower(row_seq=True): rows are (cache sequence, position) pairs, every row attends to the rows of its sequence that the same
    step writes; rows with a negative position are idle, rows marked with bit 30 want no logits (those that do come first)"""
    from oracle import gpt2_numpy as O
    from vesta_gpu_b200.launch import Kernel, TORCH_DT
    from vesta_gpu_b200.lower import lower
    from vesta_gpu_b200.program_text import decode_program
    from vesta_gpu_b200.shapes import TINY3 as sh
    rows, lens, tmax = 20, (5, 1, 11), 16
    toks = np.random.RandomState(1).randint(0, sh.N, (3, 11)).astype(np.int32)
    m, hf = model(sh, 11, 'rich', 3, tmax)
    pairs = sorted(((s, p) for s in range(3) for p in range(lens[s])), key=lambda e: e[1] != lens[e[0]] - 1)
    x, t, seq = np.zeros(rows, np.int32), np.full(rows, -1, np.int32), np.full(rows, 1 << 30, np.int32)
    for r, (s, p) in enumerate(pairs):
        x[r], t[r], seq[r] = toks[s, p], p, s | (0 if p == lens[s] - 1 else 1 << 30)
    up = lambda a: torch.from_numpy(a).cuda()
    R = {'x': up(x), 't': up(t), **m.W, 'keys': m.keys, 'vals': m.vals}
    names = {v: k for k, v in TORCH_DT.items()}
    low = lower(decode_program(sh), {n: (tuple(v.shape), names[v.dtype]) for n, v in R.items()}, {'s': tmax}, batch=rows, per_token=('x', 'keys', 'vals', 't'),
                outputs=('logit', 'next'), grid=m.k.sms, row_seq=True)
    k = Kernel(low)
    assert not k.chain
    k.bind(dict(R, row_seq=up(seq)))
    k.launch()
    k.check()
    W = O.upcast(hf.weights)
    for r, (s, _) in enumerate(pairs[:3]):
        ck, cv = O.new_cache(sh, tmax)
        for p in range(lens[s]):
            ref, nx = O.step(sh, W, ck, cv, int(toks[s, p]), p)
        assert np.abs(k.view('logit')[r].cpu().numpy() - ref).max() < 2 * TIGHT, s
        assert O.margin(ref) <= MARGIN or int(k.view('next')[r]) == nx
        for got, want in ((m.keys, ck), (m.vals, cv)):
            assert np.abs(got[s].float().cpu().numpy() - want.astype(np.float32)).max() <= 4e-3, s
