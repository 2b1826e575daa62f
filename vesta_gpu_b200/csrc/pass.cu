// Host side of the forward pass over rows (pass_kernels.cuh): sizes, workspace, tensor maps, the launches of a pass and,
// for decode steps, the CUDA graph that holds them.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <string>
#include <vector>

#include "pass_kernels.cuh"
#include "rt_internal.h"
#include "vesta_b200.h"

using namespace vesta_pass;
using vesta_rt::fail;

namespace {

int cuda_fail(cudaError_t e, const char* what) { return fail((int)e, std::string(what) + ": " + cudaGetErrorString(e)); }
#define TRY(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_fail(e_, #x); } while (0)

int up(long long v, int a) { return (int)((v + a - 1) / a * a); }

enum Kind { K_QKV = 0, K_PROJ = 1, K_FC = 2, K_P2 = 3, K_LOGITS = 4 };

struct Tile { int bm, bn, stages, splits; };

struct Layout {
    size_t z, q, act, att, gelu, part, fin, best, rowoff, pos, skip;
    size_t meta, total;                        // prompts: tokens, positions, sequences of the rows; attention runs; rows that want logits and where they go; lengths
};
// the metadata of a pass over prompts, as offsets in 32-bit words
struct Meta {
    int x, t, seq, tiles, want, dst, lens, words, max_tiles;
    Meta(int rows, int lrows, int seqs) {
        max_tiles = rows / 64 + std::min(rows, seqs) + 1;
        tiles = 0; dst = tiles + 4 * max_tiles; x = dst + 2 * lrows; t = x + rows; seq = t + rows; want = seq + rows; lens = want + lrows; words = lens + seqs;
    }
};

struct Pass {
    vesta_pass_desc d;
    int rp;                                    // rows of an operand plane when head and remainder are kept, else 0
    int planes;                                // operand rows: rp * 2, or the rows rounded up to whole tiles
    int fplanes;                               // the same for the rows that want logits
    Layout o;
    unsigned char* ws;
    Tile tile[5];
    CUtensorMap w[5], a[5];                    // weights and operand of every contraction
    int max_parts;
    std::vector<cudaGraphExec_t> graphs;       // decode: one step
    int sms;
    int* host;                                 // prompts: pinned metadata, one copy per pass of a call, then a status word
    size_t host_words;
};

// rows of an operand: one product column per row; up to 16 rows at fp32 accuracy take two planes of 8 or 16
int plane_rows(int rows, bool exact) { return !exact ? 0 : rows <= 8 ? 8 : 16; }

// Tile sizes of a contraction of `feat` features over `kb` blocks of 64 for `rows` rows (columns of the product), from a
// model of the kernel's time in microseconds, fitted to measurements on B200 (rows 16 to 16,384, folds of 768 to 6,400,
// tiles of 16 to 256 rows; within 15 % of each):
//   BM = 64 (one tile per block, whole share of the weights in flight): 1.75 + 0.22 per stage + the operand's rows;
//   BM = 128: 2.2 + 0.0065 bn for the first fill and the last epilogue, then per block of the fold the larger of the products
//     (2 bn cycles) and the loads (340 + 0.45 bn cycles), times the tiles a block takes in turn.
// A cut fold (projections) costs its parts once more in the norm that adds them.
Tile choose(int kind, int rows, int rp, int feat, int kb, int sms) {
    Tile best = {};
    double best_t = 1e30;
    const int cols = rp ? 2 * rp : rows;
    const bool cut = kind == K_PROJ || kind == K_P2;
    for (int bm = 64; bm <= 128; bm += 64)
        for (int bn = 16; bn <= (bm == 64 ? 64 : 256); bn += 16) {
            if (rp && (bm != 64 || bn != cols)) continue;
            if (bn > 16 && bn - 16 >= cols) continue;
            const int ks = bm == 64 ? GemmShape<64>::KS : GemmShape<128>::KS;
            const int stage = bm == 64 ? GemmShape<64>::stage(bn) : GemmShape<128>::stage(bn);
            const int room = 227 * 1024 - 1024 - 1024 - bn * 32;
            const int tiles = ((feat + bm - 1) / bm) * (rp ? 1 : (rows + bn - 1) / bn);
            for (int sp = 1; sp <= (cut ? PARTS_MAX : 1); sp++) {
                Tile t;
                t.bm = bm; t.bn = bn;
                const int per = (kb + sp - 1) / sp, nst = (per + ks - 1) / ks;
                t.splits = (kb + per - 1) / per;
                if (t.splits != sp) continue;
                const int waves = (tiles * sp + sms - 1) / sms;
                t.stages = std::max(1, std::min(bm == 64 || waves == 1 ? nst : 16, room / (stage + 16)));
                double us;
                if (bm == 64) us = (1.75 + 0.22 * nst + 0.0023 * (bn - 16) * per) * waves + 0.002 * tiles * sp;
                else us = 2.2 + 0.0065 * bn + waves * per * std::max(2.0 * bn + 30, 340 + 0.45 * bn) / 1900;
                if (cut && sp > 1) us += 0.1 * sp + (sp - 1) * (double)rows * feat * 4 / 4e6;
                if (us < best_t) { best_t = us; best = t; }
            }
        }
    return best;
}

Layout layout(const Pass& p, int D, int F, int rows, int lrows) {
    Layout o{};
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t r = at; at += (bytes + 255) / 256 * 256; return r; };
    o.z = take((size_t)rows * D * 4);
    o.q = take((size_t)rows * D * 4);
    o.act = take((size_t)p.planes * D * 2);
    o.att = take((size_t)p.planes * D * 2);
    o.gelu = take((size_t)p.planes * F * 2 + 128);       // (the last block of the fold may reach past the last row)
    o.part = take((size_t)p.max_parts * rows * D * 4);
    o.fin = take((size_t)p.fplanes * D * 2);
    o.best = take((size_t)lrows * 8);
    o.rowoff = take((size_t)rows * 8);
    o.pos = take((size_t)rows * 4);
    o.skip = take(4);
    o.meta = p.d.prompts ? take((size_t)Meta(rows, lrows, p.d.prompts).words * 4) : 0;
    o.total = at;
    return o;
}

int plan(Pass& p, const vesta_pass_desc* d) {
    if (!d || d->rows < 1 || d->logit_rows < 1 || d->logit_rows > d->rows) return fail(-1, "vesta_pass: bad row counts");
    if (d->L < 1 || d->D % 64 || d->D > 4096 || d->H * 64 != d->D || d->F % 16 || d->N < 1) return fail(-1, "vesta_pass: sizes outside the supported family");
    if (d->exact && d->rows > 16) return fail(-1, "vesta_pass: fp32-accurate operands are kept for at most 16 rows");
    p.d = *d;
    int dev = 0;
    p.sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&p.sms, cudaDevAttrMultiProcessorCount, dev);
    cudaGetLastError();                          // (sizes can be asked for without a device)
    p.rp = plane_rows(d->rows, d->exact != 0);
    const int frp = plane_rows(d->logit_rows, d->exact != 0);
    p.planes = p.rp ? 2 * p.rp : up(d->rows, 128);
    p.fplanes = p.rp ? 2 * p.rp : up(d->logit_rows, 128);
    (void)frp;
    const int kbd = d->D / 64, kbf = (d->F + 63) / 64;
    p.tile[K_QKV] = choose(K_QKV, d->rows, p.rp, 3 * d->D, kbd, p.sms);
    p.tile[K_PROJ] = choose(K_PROJ, d->rows, p.rp, d->D, kbd, p.sms);
    p.tile[K_FC] = choose(K_FC, d->rows, p.rp, d->F, kbd, p.sms);
    p.tile[K_P2] = choose(K_P2, d->rows, p.rp, d->D, kbf, p.sms);
    p.tile[K_LOGITS] = choose(K_LOGITS, d->logit_rows, p.rp, d->N, kbd, p.sms);
    p.max_parts = std::max(p.tile[K_PROJ].splits, p.tile[K_P2].splits);
    p.o = layout(p, d->D, d->F, d->rows, d->logit_rows);
    return 0;
}

// The kernels of a pass ask for the same split of an SM between shared memory and cache: an SM changes it only when it is idle,
// and a block that waits for that cannot start under its predecessor (23 sequences: projection 3.0 -> 2.4 us, norm 4.5 -> 3.5).
template <class F> cudaError_t all_shared(F* f) { return cudaFuncSetAttribute((const void*)f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared); }
cudaError_t prepare_all() {
    cudaError_t e = cudaSuccess;
    auto one = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    one(all_shared(pass_norm<NORM_EMBED>)); one(all_shared(pass_norm<NORM_MID>)); one(all_shared(pass_norm<NORM_FINAL>));
    one(all_shared(pass_norm_rows<6>)); one(all_shared(pass_norm_rows<13>)); one(all_shared(pass_norm_rows<16>));
    one(all_shared(pass_attend<2>)); one(all_shared(pass_attend<4>)); one(all_shared(pass_attend_many));
    one(cudaFuncSetAttribute((const void*)pass_attend<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * ATT_WARPS * 4096)); one(all_shared(pass_finish));
    return e;
}
template <int BM, int EPI>
cudaError_t launch_gemm(cudaLaunchConfig_t& c, const Tile& t, const CUtensorMap& w, const CUtensorMap& a, const GemmArgs& g) {
    c.dynamicSmemBytes = GemmShape<BM>::bytes(t.stages, t.bn);
    c.blockDim = dim3(GemmShape<BM>::THREADS);
    return cudaLaunchKernelEx(&c, pass_gemm<BM, EPI>, w, a, g);
}
template <int BM, int EPI>
cudaError_t prepare_gemm(const Tile& t) {
    const cudaError_t e = all_shared(pass_gemm<BM, EPI>);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(pass_gemm<BM, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}
// one case per tile shape and epilogue
#define EACH(X) X(64, EPI_ADD) X(128, EPI_ADD) X(64, EPI_QKV) X(64, EPI_PART) X(64, EPI_GELU) X(64, EPI_LOGITS) X(128, EPI_QKV) X(128, EPI_PART) X(128, EPI_GELU) X(128, EPI_LOGITS)
cudaError_t gemm(int epi, const Tile& t, cudaLaunchConfig_t c, const CUtensorMap& w, const CUtensorMap& a, const GemmArgs& g) {
#define ONE(M, E) if (epi == E && t.bm == M) return launch_gemm<M, E>(c, t, w, a, g);
    EACH(ONE)
#undef ONE
    return cudaErrorInvalidValue;
}
cudaError_t gemm_prepare(int epi, const Tile& t) {
#define ONE(M, E) if (epi == E && t.bm == M) return prepare_gemm<M, E>(t);
    EACH(ONE)
#undef ONE
    return cudaErrorInvalidValue;
}
int epi_of(int kind, const Tile& t) { return kind == K_QKV ? EPI_QKV : kind == K_FC ? EPI_GELU : kind == K_LOGITS ? EPI_LOGITS : t.splits > 1 ? EPI_PART : EPI_ADD; }

// launch attributes: `dependent` = may start while the kernel before it runs
struct Config {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at[2];
    Config(dim3 grid, int block, cudaStream_t st, bool dependent, int cluster = 1) {
        c.gridDim = grid; c.blockDim = dim3(block); c.stream = st; c.attrs = at; c.numAttrs = 0;
        if (dependent) { at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[c.numAttrs].val.programmaticStreamSerializationAllowed = 1; c.numAttrs++; }
        if (cluster > 1) { at[c.numAttrs].id = cudaLaunchAttributeClusterDimension; at[c.numAttrs].val.clusterDim.x = 1; at[c.numAttrs].val.clusterDim.y = 1; at[c.numAttrs].val.clusterDim.z = cluster; c.numAttrs++; }
    }
};

// The launches of one pass over `rows` rows. Prompts: `tiles` runs of rows for the attention, `lrows` rows that want logits
// (none: the pass ends with the last layer's cache rows); `clear`: zero the cache rows after the prompts.
int enqueue(Pass& p, cudaStream_t st, int rows, int lrows, int tiles, bool clear = false) {
    const vesta_pass_desc& d = p.d;
    const int D = d.D, F = d.F, L = d.L, kbd = D / 64, kbf = (F + 63) / 64;
    const bool many = d.prompts != 0;
    auto u = [&](size_t off) { return p.ws + off; };
    const Meta mt(d.rows, d.logit_rows, d.prompts);
    const int* meta = (const int*)u(p.o.meta);
    float* z = (float*)u(p.o.z);
    u16 *act = (u16*)u(p.o.act), *att = (u16*)u(p.o.att), *fin = (u16*)u(p.o.fin);
    const int nthr = up(D / 4, 32);
    auto f16 = [](const void* q, size_t off) { return (const u16*)q + off; };
    auto norm = [&](int mode, int l, int nparts) {
        NormArgs n = {};
        n.D = D; n.nparts = nparts; n.rp = p.rp; n.eps = d.eps; n.z = z;
        n.part = (const float*)u(p.o.part); n.part_stride = (size_t)d.rows * D;
        n.x = many ? meta + mt.x : (const int*)d.x; n.t = many ? meta + mt.t : (const int*)d.t; n.seq = many ? meta + mt.seq : 0; n.t_stride = many ? 1 : d.t_stride; n.N = d.N; n.cpos = d.cpos; n.tmax = d.tmax; n.L = L;
        n.wte = (const u16*)d.wte; n.wpe = (const u16*)d.wpe;
        n.rowoff = (long long*)u(p.o.rowoff); n.pos = (int*)u(p.o.pos); n.skip = (int*)u(p.o.skip); n.bar = (u32*)d.bar;
        n.want = many ? meta + mt.want : 0;
        n.act = act;
        if (mode == 0) { n.gain = f16(d.ln1w, 0); n.shift = f16(d.ln1b, 0); }
        else if (mode == 1) { n.gain = f16(d.ln2w, (size_t)l * D); n.shift = f16(d.ln2b, (size_t)l * D); n.bias = f16(d.ob, (size_t)l * D); }
        else if (mode == 2) { n.gain = f16(d.ln1w, (size_t)(l + 1) * D); n.shift = f16(d.ln1b, (size_t)(l + 1) * D); n.bias = f16(d.pb, (size_t)l * D); }
        else { n.gain = f16(d.lnfw, 0); n.shift = f16(d.lnfb, 0); n.bias = f16(d.pb, (size_t)l * D); n.act = fin; }
        if ((mode == 1 || mode == 2) && rows >= 2048 && D <= 2048 && !p.rp) {
            Config c(dim3((rows + 7) / 8), 256, st, true);
            return D <= 768 ? cudaLaunchKernelEx(&c.c, pass_norm_rows<6>, n, rows) : D <= 1664 ? cudaLaunchKernelEx(&c.c, pass_norm_rows<13>, n, rows) : cudaLaunchKernelEx(&c.c, pass_norm_rows<16>, n, rows);
        }
        Config c(dim3(mode == 3 ? lrows : rows), nthr, st, mode != 0);
        return mode == 0 ? cudaLaunchKernelEx(&c.c, pass_norm<NORM_EMBED>, n) : mode == 3 ? cudaLaunchKernelEx(&c.c, pass_norm<NORM_FINAL>, n) : cudaLaunchKernelEx(&c.c, pass_norm<NORM_MID>, n);
    };
    auto mul = [&](int kind, int l) {
        const Tile& t = p.tile[kind];
        GemmArgs g = {};
        g.layer = l; g.D = D; g.rp = p.rp; g.stages = t.stages; g.status = (u32*)d.bar; g.skip = (const int*)u(p.o.skip);
        g.rows = kind == K_LOGITS ? lrows : rows;
        g.kblocks = kind == K_P2 ? kbf : kbd; g.kb_per = (g.kblocks + t.splits - 1) / t.splits;
        g.nfeat = kind == K_QKV ? 3 * D : kind == K_FC ? F : kind == K_LOGITS ? d.N : D;
        if (kind == K_QKV) {
            g.bias = f16(d.qkvb, (size_t)l * 3 * D); g.of = (float*)u(p.o.q); g.rowoff = (const long long*)u(p.o.rowoff);
            g.kc = (u16*)d.keys + (size_t)l * d.tmax * D; g.vc = (u16*)d.vals + (size_t)l * d.tmax * D;
        } else if (kind == K_FC) {
            g.bias = f16(d.fcb, (size_t)l * F); g.oh = (u16*)u(p.o.gelu); g.a2 = 2 * d.gelu_a; g.k1 = d.gelu_b * 2.8853900817779268f; g.k2 = d.gelu_c * g.k1;
        } else if (kind == K_LOGITS) { g.of = (float*)d.logits; g.best = (u64*)u(p.o.best); }
        else if (t.splits > 1) { g.of = (float*)u(p.o.part); g.part_stride = (size_t)d.rows * D; }
        else { g.of = z; g.bias = kind == K_PROJ ? f16(d.ob, (size_t)l * D) : f16(d.pb, (size_t)l * D); }
        g.bn = t.bn; g.ftiles = (g.nfeat + t.bm - 1) / t.bm; g.rtiles = p.rp ? 1 : (g.rows + t.bn - 1) / t.bn; g.ntiles = g.ftiles * g.rtiles * t.splits;
        Config c(dim3(t.bm == 64 && kind != K_LOGITS ? g.ntiles : std::min(g.ntiles, p.sms)), 192, st, true);
        return gemm(epi_of(kind, t), t, c.c, p.w[kind], p.a[kind], g);
    };
    auto attend = [&](int l, int tiles) {
        const float* q = (const float*)u(p.o.q);
        const u16 *kc = (const u16*)d.keys + (size_t)l * d.tmax * D, *vc = (const u16*)d.vals + (size_t)l * d.tmax * D;
        const long long ss = (long long)L * d.tmax * D;
        int e = 0;
        const int pow2 = frexpf(d.scale, &e) == 0.5f;
        if (many) {
            const int zb = clear ? (2 * p.sms + d.H - 1) / d.H : 0;
            AttManyArgs a = {q, kc, vc, ss, (const int4*)(meta + mt.tiles), D, pow2, d.scale, att, zb, d.prompts, d.tmax, meta + mt.lens};
            Config c(dim3(zb + tiles, d.H), 128, st, true);
            return cudaLaunchKernelEx(&c.c, pass_attend_many, a);
        }
        AttArgs a = {q, kc, vc, ss, (const int*)d.t, (const int*)0, d.t_stride, d.tmax, D, pow2, p.rp, d.scale, att};
        int C = 1;
        while (C < 8 && rows * d.H * C * 2 <= 6 * p.sms && d.tmax > C * ATT_WARPS * ATT_RUN) C *= 2;
        Config c(dim3(d.H, rows, C), ATT_WARPS * 32, st, true, C);
        // deep rings where few blocks share an SM, all blocks resident where they are many
        const bool deep = rows * d.H * C <= 3 * p.sms;
        c.c.dynamicSmemBytes = (deep ? 4 : 2) * ATT_WARPS * 4096;
        return deep ? cudaLaunchKernelEx(&c.c, pass_attend<4>, a) : cudaLaunchKernelEx(&c.c, pass_attend<2>, a);
    };
    TRY(norm(0, 0, 0));
    for (int l = 0; l < L; l++) {
        TRY(mul(K_QKV, l));
        const bool end = l == L - 1 && lrows == 0;
        if (!end || clear) TRY(attend(l, end ? 0 : tiles));
        if (end) break;
        TRY(mul(K_PROJ, l));
        TRY(norm(1, l, p.tile[K_PROJ].splits > 1 ? p.tile[K_PROJ].splits : 0));
        TRY(mul(K_FC, l));
        TRY(mul(K_P2, l));
        TRY(norm(l + 1 < L ? 2 : 3, l, p.tile[K_P2].splits > 1 ? p.tile[K_P2].splits : 0));
    }
    if (lrows) TRY(mul(K_LOGITS, 0));
    FinishArgs f = {};
    f.rows = lrows; f.best = (u64*)u(p.o.best); f.skip = (int*)u(p.o.skip); f.next = (float*)d.next; f.pos = (const int*)u(p.o.pos);
    f.t_stride = d.t_stride; f.tstep = d.tstep; f.N = d.N;
    if (many) { f.dst = (const int2*)(meta + mt.dst); f.x = (int*)d.x; f.t = (int*)d.t; }
    else if (d.feedback) { f.x = (int*)d.x; f.t = (int*)d.t; f.prompt = (const int*)d.prompt; f.plen = (const int*)d.plen; f.plen_cap = d.prompt_len; }
    Config c(dim3(1), 256, st, true);
    TRY(cudaLaunchKernelEx(&c.c, pass_finish, f));
    return 0;
}

}  // namespace

namespace vesta_rt {
int pass_steps(void* pass, void* stream, int steps) {
    Pass* p = (Pass*)pass;
    cudaStream_t st = (cudaStream_t)stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TRY(cudaStreamIsCapturing(st, &cap));
    for (int i = 0; i < steps; i++) {
        if (cap != cudaStreamCaptureStatusNone || p->graphs.empty()) { if (int e = enqueue(*p, st, p->d.rows, p->d.logit_rows, 0)) return e; }
        else TRY(cudaGraphLaunch(p->graphs[0], st));
    }
    return 0;
}
}  // namespace vesta_rt

extern "C" {

int vesta_pass_workspace(const vesta_pass_desc* d, size_t* bytes) {
    Pass p{};
    if (!bytes) return fail(-1, "vesta_pass_workspace: null argument");
    if (int e = plan(p, d)) return e;
    *bytes = p.o.total;
    return 0;
}

int vesta_pass_create(const vesta_pass_desc* d, void* workspace, int graph, void** out) {
    if (!out || !workspace) return fail(-1, "vesta_pass_create: null argument");
    Pass* p = new Pass{};
    int e = plan(*p, d);
    p->ws = (unsigned char*)workspace;
    const int D = d->D, F = d->F;
    const void* w[5] = {d->qkvw, d->ow, d->fcw, d->pw, d->wte};
    const int fold[5] = {D, D, D, F, D}, feat[5] = {3 * D, D, F, D, d->N};
    if (!e) { const cudaError_t ce = prepare_all(); if (ce != cudaSuccess) e = cuda_fail(ce, "cudaFuncSetAttribute"); }
    unsigned char* op[5] = {p->ws + p->o.act, p->ws + p->o.att, p->ws + p->o.act, p->ws + p->o.gelu, p->ws + p->o.fin};
    for (int k = 0; k < 5 && !e; k++) {
        const Tile& t = p->tile[k];
        const int ks = t.bm == 64 ? GemmShape<64>::KS : GemmShape<128>::KS;
        if (k == K_LOGITS) e = vesta_rt::fold_map(&p->w[k], w[k], D, feat[k], t.bm, ks);
        else e = vesta_rt::tensor_map(&p->w[k], w[k], feat[k], fold[k], d->L, (size_t)feat[k] * 2, (size_t)feat[k] * fold[k] * 2, 64 * ks, 1);
        if (!e) e = vesta_rt::fold_map(&p->a[k], op[k], fold[k], k == K_LOGITS ? p->fplanes : p->planes, t.bn, ks);
        if (!e) { const cudaError_t ce = gemm_prepare(epi_of(k, p->tile[k]), p->tile[k]); if (ce != cudaSuccess) e = cuda_fail(ce, "cudaFuncSetAttribute"); }
    }
    if (!e && graph) {
        // a decode step as a graph, captured on a stream of its own
        cudaStream_t st = nullptr;
        cudaGraph_t g = nullptr;
        cudaGraphExec_t ge = nullptr;
        cudaError_t ce = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (ce == cudaSuccess) ce = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
        if (ce == cudaSuccess) {
            e = enqueue(*p, st, d->rows, d->logit_rows, 0);
            ce = cudaStreamEndCapture(st, &g);
        }
        if (ce == cudaSuccess && !e) ce = cudaGraphInstantiate(&ge, g, 0);
        if (ge) p->graphs.push_back(ge);
        if (g) cudaGraphDestroy(g);
        if (st) cudaStreamDestroy(st);
        if (ce != cudaSuccess && !e) e = cuda_fail(ce, "vesta_pass_create: graph of a step");
    }
    if (e) { vesta_pass_release(p); return e; }
    *out = p;
    return 0;
}

int vesta_pass_prompts(void* pass, void* stream, const int* tokens, int ld, const int* lens, unsigned* status) {
    Pass* p = (Pass*)pass;
    if (!p || !p->d.prompts || !tokens || !lens || !status) return fail(-1, "vesta_pass_prompts: bad argument");
    const vesta_pass_desc& d = p->d;
    cudaStream_t st = (cudaStream_t)stream;
    const int B = d.prompts;
    const Meta mt(d.rows, d.logit_rows, B);
    long long total = 0;
    for (int s = 0; s < B; s++) {
        if (lens[s] < 1 || lens[s] > ld || lens[s] > d.tmax) return fail(-1, "vesta_pass_prompts: a prompt length is outside 1 .. tmax");
        total += lens[s];
    }
    // passes of equal size (whole tiles of 128 rows): two of 9,200 rows rather than one of 16,384 and a small one
    const int passes = (int)((total + d.rows - 1) / d.rows);
    const int per = std::min<long long>(d.rows, up((total + passes - 1) / passes, 128));
    const size_t words = (size_t)passes * mt.words + 4;
    if (p->host_words < words) {
        if (p->host) cudaFreeHost(p->host);
        p->host = nullptr; p->host_words = 0;
        TRY(cudaMallocHost((void**)&p->host, words * 4));
        p->host_words = words;
    }
    struct Run { int first, rows, seq, pos; };
    std::vector<Run> runs;
    int s = 0, pos = 0;                          // next position to read
    for (int c = 0; c < passes; c++) {
        int* m = p->host + (size_t)c * mt.words;
        int n = 0, lrows = 0;
        runs.clear();
        while (n < per && s < B) {
            const int take = std::min(per - n, lens[s] - pos);
            for (int i = 0; i < take; i++) { m[mt.x + n + i] = tokens[(size_t)s * ld + pos + i]; m[mt.t + n + i] = pos + i; m[mt.seq + n + i] = s; }
            for (int i = 0; i < take; i += 64) runs.push_back(Run{n + i, std::min(64, take - i), s, pos + i});
            n += take; pos += take;
            if (pos == lens[s]) {
                m[mt.want + lrows] = n - 1; m[mt.dst + 2 * lrows] = s; m[mt.dst + 2 * lrows + 1] = lens[s];
                lrows++; s++; pos = 0;
            }
        }
        // the runs that see most positions first
        std::stable_sort(runs.begin(), runs.end(), [](const Run& a, const Run& b) { return a.pos + a.rows > b.pos + b.rows; });
        for (size_t i = 0; i < runs.size(); i++) { int* t = m + mt.tiles + 4 * i; t[0] = runs[i].first; t[1] = runs[i].rows; t[2] = runs[i].seq; t[3] = runs[i].pos; }
        for (int i = 0; i < B; i++) m[mt.lens + i] = lens[i];
        TRY(cudaMemcpyAsync(p->ws + p->o.meta, m, (size_t)mt.words * 4, cudaMemcpyHostToDevice, st));
        if (int e = enqueue(*p, st, n, lrows, (int)runs.size(), c == 0)) return e;
    }
    unsigned* word = (unsigned*)(p->host + words - 4);
    TRY(cudaMemcpyAsync(word, d.bar, 4, cudaMemcpyDeviceToHost, st));
    TRY(cudaStreamSynchronize(st));
    *status = *word;
    return 0;
}

void vesta_pass_release(void* pass) {
    Pass* p = (Pass*)pass;
    if (!p) return;
    for (auto g : p->graphs) cudaGraphExecDestroy(g);
    if (p->host) cudaFreeHost(p->host);
    delete p;
}

}  // extern "C"
