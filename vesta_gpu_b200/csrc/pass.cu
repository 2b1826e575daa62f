// Host side of the forward pass over rows (pass_kernels.cuh): sizes, workspace, tensor maps, the launches of a pass and,
// for decode steps, the CUDA graph that holds them.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <exception>
#include <string>
#include <vector>

#include "pass_few.cuh"
#include "pass_kernels.cuh"
#include "rt_internal.h"
#include "vesta_b200.h"

using namespace vesta_pass;
using vesta_rt::fail;

namespace {

int cuda_fail(cudaError_t e, const char* what) { return fail((int)e, std::string(what) + ": " + cudaGetErrorString(e)); }
#define TRY(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) return cuda_fail(e_, #x); } while (0)

int up(long long v, int a) { return (int)((v + a - 1) / a * a); }

const u64 WAIT_NS = 500000000ull;              // waits of a new pass give up after half a second

enum Kind { K_QKV = 0, K_PROJ = 1, K_FC = 2, K_P2 = 3, K_LOGITS = 4 };

struct Tile { int bm, bn, stages, splits; };

struct Layout {
    size_t z, q, act, att, gelu, fin, best, rowoff, pos, skip;
    size_t after[2], sums[2], packed;          // few sequences: the state after the attention and the MLP's sums, of two layers in turn; the packed weights
    size_t meta, total;                        // prompts: tokens, positions, sequences of the rows; attention runs; rows that want logits and where they go; lengths
};
// the metadata of a pass over prompts, as offsets in 32-bit words
struct Meta {
    int x, t, seq, tiles, want, dst, lens, words, max_tiles;
    Meta(int rows, int lrows, int seqs) {
        max_tiles = rows / 128 + std::min(rows, seqs) + 1;
        tiles = 0; dst = tiles + 4 * max_tiles; x = dst + 2 * lrows; t = x + rows; seq = t + rows; want = seq + rows; lens = want + lrows; words = lens + seqs;
    }
};

// A decode step of few sequences (pass_few.cuh): tiles per block of the two kernels that cut features
struct Few {
    bool on, fixed;                            // fixed: the state as State<true>, and four warps to a row instead of two
    int qkv_per, mlp_per;
};
const int SMEM_MAX = 227 * 1024;

struct Pass {
    vesta_pass_desc d;
    Few few;
    int rp;                                    // rows of an operand plane when head and remainder are kept, else 0
    int planes;                                // operand rows: rp * 2, or the rows rounded up to whole tiles
    int fplanes;                               // the same for the rows that want logits
    Layout o;
    unsigned char* ws;
    struct Plan {                              // tiles for a number of rows
        int rows, lrows;
        Tile tile[5];
        CUtensorMap w[5], a[5];                // weights and operand of every contraction
    };
    std::vector<Plan> plans;                   // the last few
    CUtensorMap qmap, kmap, vmap;              // prompts: queries (two planes) and the caches, 128 rows of one head per box
    cudaGraphExec_t graph;                     // decode: one step, or null
    int sms, dev;
    u64 wait_ns;                               // limit of a wait
    int* host;                                 // prompts: pinned metadata, one copy per pass of a call, then a status word
    size_t host_words;
};

// rows of an operand: one product column per row; up to 16 rows at fp32 accuracy take two planes of 8 or 16
int plane_rows(int rows, bool exact) { return !exact ? 0 : rows <= 8 ? 8 : 16; }

// Tile sizes of a contraction of `feat` features over `kb` blocks of 64 for `rows` rows (columns of the product), from a
// model of the kernel's time in microseconds, fitted to measurements on B200 (rows 16 to 16,384, folds of 768 to 6,400,
// tiles of 16 to 256 rows) of a kernel by itself, its weights in L2: within 15 % of each. It ranks tiles; it is not the time of a
// kernel in a pass, where its boundary and weights that come from memory are added (9,200 rows of the small shape, FC: 36.5
// and 38.3 seen, QKV 26.5 and 31.7; 77 rows, QKV 3.1 and 4.5; 16 of the XL shape, QKV 4.4 and 4.5, MLP projection 3.2 and 6.1):
//   BM = 64 (one tile per block, whole share of the weights in flight): 1.75, 0.22 per stage, 0.5 for every stage that has to
//     wait for a free one, the operand's rows;
//   BM = 128: 2.2 for the first fill, a term for the last epilogue, then per block of the fold the larger of the products and the loads
//     (L2 into the SMs, the slower the more SMs take part); with several tiles per block, each but the last costs the larger
//     of that and its epilogue;
//   BM = 256 (two blocks): 3.0, and a third less for the loads: better for folds of more than about 1,000.
// A cut fold (projections) costs one more reduction per element and part: hidden by the chain up to about 0.5 MB of sums.
Tile choose(int kind, int rows, int rp, int feat, int kb, int sms) {
    Tile best = {};
    double best_t = 1e30;
    const int cols = rp ? 2 * rp : rows;
    const bool cut = kind == K_PROJ || kind == K_P2;
    const double last = kind == K_FC ? 0.012 : kind == K_QKV ? 0.009 : 0.0065;
    for (int bm = 64; bm <= 256; bm *= 2)
        for (int bn = 16; bn <= (bm == 64 ? 64 : 256); bn += 16) {
            if (rp && (bm != 64 || bn != cols)) continue;
            if ((bn > 16 && bn - 16 >= cols) || (bm == 256 && (bn < 64 || kind == K_LOGITS))) continue;
            const int ks = bm == 64 ? GemmShape<64>::KS : 1;
            const int stage = bm == 64 ? GemmShape<64>::stage(bn) : bm == 128 ? GemmShape<128>::stage(bn) : GemmShape<256>::stage(bn);
            const int room = 227 * 1024 - 1024 - 1024 - bn * 32;
            const int tiles = ((feat + bm - 1) / bm) * (rp ? 1 : (rows + bn - 1) / bn);
            const int units = bm == 256 ? sms / 2 : sms;
            const double epi = kind == K_FC || kind == K_LOGITS ? 0.016 * bn + 1.2 : kind == K_QKV ? 0.010 * bn + 2.0 : 0.0145 * bn + 1.7;
            for (int sp = 1; sp <= (cut ? PARTS_MAX : 1); sp++) {
                Tile t;
                t.bm = bm; t.bn = bn;
                const int per = (kb + sp - 1) / sp, nst = (per + ks - 1) / ks;
                t.splits = (kb + per - 1) / per;
                if (t.splits != sp) continue;
                const int waves = (tiles * sp + units - 1) / units;
                t.stages = std::max(1, std::min(bm == 64 || waves == 1 ? nst : 16, room / (stage + 16)));
                double us;
                if (bm == 64) us = (1.75 + 0.22 * nst + 0.5 * std::max(0, nst - t.stages) + 0.0023 * (bn - 16) * per) * waves + 0.002 * tiles * sp;
                else {
                    const double busy = std::min(1.0, (double)tiles * sp / (0.88 * units));
                    const double kb_us = bm == 128 ? std::max(std::max(0.0011 * bn + 0.03, 0.19), busy * (0.0016 * bn + 0.02)) : 0.0010 * bn + 0.04 + 0.033 * busy;
                    const double main = per * kb_us;
                    us = (bm == 128 ? 2.2 : 3.0) + last * bn + main + (waves - 1) * std::max(main, epi);
                }
                if (cut) {
                    const double mb = rows * (double)feat * 4e-6;
                    us += (sp - 1) * (mb < 0.5 ? 0.125 * mb : 0.13 + 0.1 * mb);
                }
                if (us < best_t) { best_t = us; best = t; }
            }
        }
    return best;
}
int k_blocks(int bm) { return bm == 64 ? GemmShape<64>::KS : 1; }
int box_rows(const Tile& t) { return t.bm == 256 ? t.bn / 2 : t.bn; }

Layout layout(const Pass& p, int D, int F, int rows, int lrows) {
    Layout o{};
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t r = at; at += (bytes + 255) / 256 * 256; return r; };
    if (p.few.on) {
        const size_t state = (size_t)rows * D * (p.few.fixed ? 8 : 4);
        for (int i = 0; i < 2; i++) { o.after[i] = take(state); o.sums[i] = take(state); }
        o.q = take((size_t)rows * D * 4);
        o.fin = take((size_t)p.fplanes * D * 2);
        o.best = take((size_t)lrows * 8);
        o.pos = take((size_t)rows * 4);
        o.skip = take(4);
        o.packed = take(FewPack(D, F).layer * p.d.L);
        o.total = at;
        return o;
    }
    o.z = take((size_t)rows * D * 4);
    o.q = take((size_t)rows * D * 4);
    o.act = take((size_t)p.planes * D * 2);
    o.att = take((size_t)p.planes * D * 2);
    o.gelu = take((size_t)p.planes * up(F, 64) * 2);     // (whole blocks of the fold per row: no product meets another row's values)
    o.fin = take((size_t)p.fplanes * D * 2);
    o.best = take((size_t)lrows * 8);
    o.rowoff = take((size_t)rows * 8);
    o.pos = take((size_t)rows * 4);
    o.skip = take(4);
    o.meta = p.d.prompts ? take((size_t)Meta(rows, lrows, p.d.prompts).words * 4) : 0;
    o.total = at;
    return o;
}

// The tiles of a step of few sequences: about a block per SM, as far as the blocks' weights fit shared memory; false: they do not, or not
// every row wants logits (the end of such a step writes a row of logits, a token and a position for each).
bool few_plan(Pass& p, const vesta_pass_desc& d) {
    if (d.rows < 2 || d.rows > FEW_ROWS || d.logit_rows != d.rows || d.prompts || d.D > 1024) return false;
    Few f{};
    f.on = true;
    f.fixed = d.rows == 2;
    const int sms = 148;
    f.qkv_per = (3 * d.D / 16 + sms - 1) / sms;
    f.mlp_per = (d.F / 16 + sms - 1) / sms;
    if (std::max(f.qkv_per, f.mlp_per) > FEW_TILES || FewMlp::bytes(d.D, d.rows, f.mlp_per) > SMEM_MAX - 1024) return false;
    p.few = f;
    return true;
}

int plan(Pass& p, const vesta_pass_desc* d) {
    if (!d || d->rows < 1 || d->rows > 1 << 28 || d->logit_rows < 1 || d->logit_rows > d->rows) return fail(-1, "vesta_pass: bad row counts");
    if (d->prompts < 0 || (d->prompts && d->logit_rows < std::min(d->rows, d->prompts))) return fail(-1, "vesta_pass: a pass over prompts needs a logit row for every prompt that can end in it");
    if (d->L < 1 || d->D < 64 || d->D % 64 || d->D > 4096 || d->H * 64 != d->D || d->F < 16 || d->F % 16 || d->N < 1 || d->tmax < 1 || d->cpos < 1) return fail(-1, "vesta_pass: sizes outside the supported family");
    p.few = Few{};
    if (d->exact == 2 && !few_plan(p, *d)) return fail(-1, "vesta_pass: sizes outside those of a step from packed weights");
    if (d->exact && d->rows > 16) return fail(-1, "vesta_pass: fp32-accurate operands are kept for at most 16 rows");
    p.d = *d;
    p.dev = 0;
    p.wait_ns = WAIT_NS;
    p.sms = 148;
    if (cudaGetDevice(&p.dev) == cudaSuccess) cudaDeviceGetAttribute(&p.sms, cudaDevAttrMultiProcessorCount, p.dev);
    cudaGetLastError();                          // (sizes can be asked for without a device)
    p.rp = plane_rows(d->rows, d->exact != 0);
    p.planes = p.rp ? 2 * p.rp : up(d->rows, 128);
    p.fplanes = p.rp ? 2 * p.rp : up(d->logit_rows, 128);
    p.o = layout(p, d->D, d->F, d->rows, d->logit_rows);
    return 0;
}

// The weights and caches are there and start where the kernels' loads want them: 16 bytes for tensor copies and 16-byte pieces, 8 for
// the norms' parameters and the position table, and for the biases that the norms of a step from packed weights start the next sums with
int check(const vesta_pass_desc& d) {
    const void* wide[] = {d.wte, d.qkvw, d.ow, d.fcw, d.pw, d.keys, d.vals};
    const void* four[] = {d.wpe, d.ln1w, d.ln1b, d.ln2w, d.ln2b, d.lnfw, d.lnfb};
    for (const void* q : {(const void*)d.qkvb, (const void*)d.ob, (const void*)d.fcb, (const void*)d.pb, (const void*)d.x, (const void*)d.t, (const void*)d.logits, (const void*)d.bar})
        if (!q) return fail(-1, "vesta_pass: a tensor is missing");
    for (const void* q : wide) if (!q || (size_t)q % 16) return fail(-1, "vesta_pass: matrices, table and caches start on a 16-byte boundary");
    for (const void* q : four) if (!q || (size_t)q % 8) return fail(-1, "vesta_pass: norm parameters and position table start on an 8-byte boundary");
    for (const void* q : {d.ob, d.pb}) if (d.exact == 2 && (size_t)q % 8) return fail(-1, "vesta_pass: for a step from packed weights the projections' biases start on an 8-byte boundary");
    return 0;
}

// The kernels of a pass ask for the same split of an SM between shared memory and cache: an SM changes it only when it is idle,
// and a block that waits for that cannot start under its predecessor (23 sequences: projection 3.0 -> 2.4 us, norm 4.5 -> 3.5).
template <class F> cudaError_t all_shared(F* f) { return cudaFuncSetAttribute((const void*)f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared); }
template <int BM, int EPI>
cudaError_t launch_gemm(cudaLaunchConfig_t& c, const Tile& t, const CUtensorMap& w, const CUtensorMap& a, const GemmArgs& g) {
    c.blockDim = dim3(GemmShape<BM>::THREADS + (EPI == EPI_QKV && g.seqs ? 32 : 0));
    return cudaLaunchKernelEx(&c, pass_gemm<BM, EPI>, w, a, g);
}
template <int BM, int EPI>
cudaError_t prepare_gemm() {
    const cudaError_t e = all_shared(pass_gemm<BM, EPI>);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(pass_gemm<BM, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}
// one case per tile shape and epilogue
#define EACH(X) X(256, EPI_ADD) X(256, EPI_QKV) X(256, EPI_GELU) X(64, EPI_ADD) X(128, EPI_ADD) X(64, EPI_QKV) X(64, EPI_GELU) X(64, EPI_LOGITS) X(128, EPI_QKV) X(128, EPI_GELU) X(128, EPI_LOGITS)
cudaError_t gemm(int epi, const Tile& t, cudaLaunchConfig_t c, const CUtensorMap& w, const CUtensorMap& a, const GemmArgs& g) {
#define ONE(M, E) if (epi == E && t.bm == M) return launch_gemm<M, E>(c, t, w, a, g);
    EACH(ONE)
#undef ONE
    return cudaErrorInvalidValue;
}
cudaError_t gemm_prepare() {
    cudaError_t e = cudaSuccess;
#define ONE(M, E) if (e == cudaSuccess) e = prepare_gemm<M, E>();
    EACH(ONE)
#undef ONE
    return e;
}
cudaError_t prepare_all() {
    cudaError_t e = cudaSuccess;
    auto one = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    one(all_shared(pass_norm<NORM_EMBED>)); one(all_shared(pass_norm<NORM_MID>)); one(all_shared(pass_norm<NORM_FINAL>));
    one(all_shared(pass_norm_rows<6>)); one(all_shared(pass_norm_rows<13>)); one(all_shared(pass_norm_rows<16>));
    one(all_shared(pass_attend<2, 4>)); one(all_shared(pass_attend<4, 4>)); one(all_shared(pass_attend<2, 8>)); one(all_shared(pass_attend<3, 8>)); one(all_shared(pass_attend_many<true>)); one(all_shared(pass_attend_many<false>));
    one(gemm_prepare());
    one(cudaFuncSetAttribute((const void*)pass_attend_many<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AM_SMEM));
    one(cudaFuncSetAttribute((const void*)pass_attend_many<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AM_SMEM));
    one(cudaFuncSetAttribute((const void*)pass_attend<3, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * 8 * 4096));
    one(cudaFuncSetAttribute((const void*)pass_attend<4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 4 * 4096));
    one(cudaFuncSetAttribute((const void*)pass_attend<2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * 8 * 4096)); one(all_shared(pass_finish));
    return e;
}
int epi_of(int kind) { return kind == K_QKV ? EPI_QKV : kind == K_FC ? EPI_GELU : kind == K_LOGITS ? EPI_LOGITS : EPI_ADD; }

// launch attributes: `dependent` = may start while the kernel before it runs (a contraction's launch sets its threads by itself)
struct Config {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at[2];
    Config(dim3 grid, int block, cudaStream_t st, bool dependent, int cluster = 1, bool along_x = false) {
        c.gridDim = grid; c.blockDim = dim3(block); c.stream = st; c.attrs = at; c.numAttrs = 0;
        if (dependent) { at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[c.numAttrs].val.programmaticStreamSerializationAllowed = 1; c.numAttrs++; }
        if (cluster > 1) { at[c.numAttrs].id = cudaLaunchAttributeClusterDimension; at[c.numAttrs].val.clusterDim.x = along_x ? cluster : 1; at[c.numAttrs].val.clusterDim.y = 1; at[c.numAttrs].val.clusterDim.z = along_x ? 1 : cluster; c.numAttrs++; }
    }
};

// the tile of contraction `k` for `rows` rows of which `lrows` want logits
Tile tile_of(const Pass& p, int k, int rows, int lrows) {
    const vesta_pass_desc& d = p.d;
    const int feat[5] = {3 * d.D, d.D, d.F, d.D, d.N};
    return choose(k, k == K_LOGITS ? std::max(lrows, 1) : rows, p.rp, feat[k], k == K_P2 ? (d.F + 63) / 64 : d.D / 64, p.sms);
}

// Shared memory of a block of a contraction of `ntiles` tiles. The projection of few rows has small blocks that come while the attention's leave: five of
// them on the first SMs that are free, none on the last. Where there is about one for every SM and more than two would fit one, they ask for
// so much that only two do (64 sequences, 144 blocks of 41 KB: 1,763 -> 1,721 us per four steps; 33 to 80 sequences 1 to 4 % faster; 23, 72 blocks:
// 1,111 -> 1,122, left). Blocks of the XL shape (83 KB) are two to an SM as they are, and with more lose their place beside an attention block
// (16 sequences at 300 positions 1,367 -> 1,355 us per step without, 8 at 300 1,309 -> 1,288), as do those of width 1,280 (16 at 128 315 -> 304).
// Short prompts gain too (77 rows 368.7 -> 366.4 us, 120 rows 408.7 -> 402.1), others take the same time (100, 200 to 900 rows).
size_t block_bytes(const Pass& p, int kind, const Tile& t, int ntiles) {
    const int bytes = t.bm == 64 ? GemmShape<64>::bytes(t.stages, t.bn) : t.bm == 128 ? GemmShape<128>::bytes(t.stages, t.bn) : GemmShape<256>::bytes(t.stages, t.bn);
    const bool spread = kind == K_PROJ && p.d.D <= 1024 && t.bm == 64 && 2 * ntiles > p.sms && 3 * (bytes + 1024) <= SMEM_MAX;
    return spread ? std::max(bytes, 110 * 1024) : bytes;
}

// The tiles and tensor maps for `rows` rows of which `lrows` want logits.
int plan_for(Pass& p, int rows, int lrows, const Pass::Plan** out) {
    for (auto& q : p.plans) if (q.rows == rows && q.lrows == lrows) { *out = &q; return 0; }
    if (p.plans.size() >= 8) p.plans.erase(p.plans.begin());
    const vesta_pass_desc& d = p.d;
    const int D = d.D, F = d.F;
    Pass::Plan q;
    q.rows = rows; q.lrows = lrows;
    const void* w[5] = {d.qkvw, d.ow, d.fcw, d.pw, d.wte};
    const int fold[5] = {D, D, D, F, D}, pitch[5] = {D, D, D, up(F, 64), D}, feat[5] = {3 * D, D, F, D, d.N};
    const size_t op[5] = {p.o.act, p.o.att, p.o.act, p.o.gelu, p.o.fin};
    for (int k = p.few.on ? K_LOGITS : 0; k < 5; k++) {             // (few sequences: of these contractions the logits only)
        const Tile t = q.tile[k] = tile_of(p, k, rows, lrows);
        int e;
        if (k == K_LOGITS) e = vesta_rt::fold_map(&q.w[k], w[k], D, feat[k], t.bm, k_blocks(t.bm));
        else e = vesta_rt::tensor_map(&q.w[k], w[k], feat[k], fold[k], d.L, (size_t)feat[k] * 2, (size_t)feat[k] * fold[k] * 2, 64 * k_blocks(t.bm), 1);
        if (!e) e = vesta_rt::fold_map(&q.a[k], p.ws + op[k], pitch[k], k == K_LOGITS ? p.fplanes : p.planes, box_rows(t), k_blocks(t.bm));
        if (e) return e;
    }
    p.plans.push_back(q);
    *out = &p.plans.back();
    return 0;
}

FinishArgs finish(const Pass& p, int lrows) {
    const vesta_pass_desc& d = p.d;
    FinishArgs f = {};
    f.rows = lrows; f.best = (u64*)(p.ws + p.o.best); f.skip = (int*)(p.ws + p.o.skip); f.bar = (const u32*)d.bar; f.next = (float*)d.next; f.pos = (const int*)(p.ws + p.o.pos);
    f.t_stride = d.t_stride; f.tstep = d.tstep; f.N = d.N;
    if (d.feedback && !d.prompts) { f.x = (int*)d.x; f.t = (int*)d.t; f.prompt = (const int*)d.prompt; f.plen = (const int*)d.plen; f.plen_cap = d.prompt_len; }
    return f;
}
GemmArgs logits_args(const Pass& p, const Tile& t, int lrows) {
    GemmArgs g = {};
    g.D = p.d.D; g.rp = p.rp; g.stages = t.stages; g.status = (u32*)p.d.bar; g.limit = p.wait_ns; g.skip = (const int*)(p.ws + p.o.skip);
    g.rows = lrows; g.kblocks = p.d.D / 64; g.kb_per = g.kblocks; g.nfeat = p.d.N;
    g.of = (float*)p.d.logits; g.best = (u64*)(p.ws + p.o.best);
    g.bn = t.bn; g.ftiles = (g.nfeat + t.bm - 1) / t.bm; g.rtiles = p.rp ? 1 : (g.rows + t.bn - 1) / t.bn; g.ntiles = g.ftiles * g.rtiles * t.splits;
    return g;
}

// The launches of one pass over `rows` rows. Prompts: `tiles` runs of rows for the attention, `lrows` rows that want logits
// (none: the pass ends with the last layer's cache rows); `clear`: zero the cache rows behind the ones that the pass writes.
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
    // attention of a step: two blocks per (row, head) where that is at most three blocks per SM and the cache has two runs of
    // positions. Clusters of four and eight lost everywhere (XL shape, 6 sequences at 128 positions: 1,342 -> 1,337 us per
    // step with two blocks instead of four; 9 sequences, small shape, two instead of eight: 298 -> 270 us, at 1,000 positions
    // 340 -> 321), and so did two beyond that line (23 sequences at 128 positions with one block: 294 -> 277 us).
    const int C = rows * d.H * 2 <= 3 * p.sms && d.tmax > 4 * ATT_RUN ? 2 : 1;
    // Warps and stages of a block's rings. Where two blocks are due to an SM, eight warps and 96 KB, which keep a third block away: blocks
    // go where there is room, which is not evenly (23 ragged sequences to 700 positions: 7.05 us with 4 x 4, 4.92 so; 9 at 900: 290 and 272 us per
    // step, at 8 positions 244 and 239). Not so: clusters of two that nearly fill the SMs, whose last ones wait until both their places are
    // free (12 sequences at 64 positions 242 us per step with 4 x 4, 248 so); wide rows with fewer blocks, where an SM with two of them
    // has no room for the projection's block of 83 KB, which 64 KB leave (XL shape, 4 at 64: 1,149 and 1,239, 9 at 64: 1,208 and 1,223; with 10
    // and 11, one for nearly every place, it is 0.99 to 1.06 times as fast). Elsewhere up to three blocks per SM four warps with 64 KB, which is
    // within 1 % of eight with 64 from 300 positions and up to 2 % faster below, but for wide rows of one block per pair, where eight are 1 to 2 %
    // faster from 64 positions (XL shape, 16 at 300: 1,372 and 1,357; at 8 1,174 and 1,185). Beyond, 32 KB: 64 sequences 16.0 us, with eight warps 17.1.
    // How blocks of several kernels share an SM depends on the width: all this holds at widths of 640 to 1,024 and from 1,600 on. Width 512 loses in
    // clusters of two (14 sequences at 64 positions 229 us per step with 4 x 4, 240 with eight warps and 96 KB), 1,280 with eight warps of either kind (13 at 128:
    // 294 and 308, 16 at 128: 301 and 305): four warps there.
    const int blocks = rows * d.H * C;
    const bool narrow = D <= 1024, wide = D >= 1536, some = blocks <= 3 * p.sms;
    const bool deep = (narrow && 4 * blocks > 5 * p.sms) || (wide && 8 * blocks > 13 * p.sms);
    const int shape = deep && (C == 2 ? D > 512 && 10 * blocks <= 17 * p.sms : blocks <= 2 * p.sms) ? 83 : !some ? 42 : wide && C == 1 ? 82 : 44;
    const Pass::Plan* pl = nullptr;
    if (int e = plan_for(p, rows, lrows, &pl)) return e;
    auto f16 = [](const void* q, size_t off) { return (const u16*)q + off; };
    auto norm = [&](int mode, int l) {
        NormArgs n = {};
        n.D = D; n.rp = p.rp; n.eps = d.eps; n.z = z;
        n.x = many ? meta + mt.x : (const int*)d.x; n.t = many ? meta + mt.t : (const int*)d.t; n.seq = many ? meta + mt.seq : 0; n.t_stride = many ? 1 : d.t_stride; n.N = d.N; n.cpos = d.cpos; n.tmax = d.tmax; n.L = L;
        n.wte = (const u16*)d.wte; n.wpe = (const u16*)d.wpe;
        n.rowoff = (long long*)u(p.o.rowoff); n.pos = (int*)u(p.o.pos); n.skip = (int*)u(p.o.skip); n.bar = (u32*)d.bar;
        n.want = many ? meta + mt.want : 0;
        n.act = act;
        if (mode == 0) { n.gain = f16(d.ln1w, 0); n.shift = f16(d.ln1b, 0); }
        else if (mode == 1) { n.gain = f16(d.ln2w, (size_t)l * D); n.shift = f16(d.ln2b, (size_t)l * D); }
        else if (mode == 2) { n.gain = f16(d.ln1w, (size_t)(l + 1) * D); n.shift = f16(d.ln1b, (size_t)(l + 1) * D); }
        else { n.gain = f16(d.lnfw, 0); n.shift = f16(d.lnfb, 0); n.act = fin; }
        if ((mode == 1 || mode == 2) && rows >= 2048 && D <= 2048 && !p.rp) {
            Config c(dim3((rows + 7) / 8), 256, st, true);
            return D <= 768 ? cudaLaunchKernelEx(&c.c, pass_norm_rows<6>, n, rows) : D <= 1664 ? cudaLaunchKernelEx(&c.c, pass_norm_rows<13>, n, rows) : cudaLaunchKernelEx(&c.c, pass_norm_rows<16>, n, rows);
        }
        Config c(dim3(mode == 3 ? lrows : rows), nthr, st, mode != 0);
        return mode == 0 ? cudaLaunchKernelEx(&c.c, pass_norm<NORM_EMBED>, n) : mode == 3 ? cudaLaunchKernelEx(&c.c, pass_norm<NORM_FINAL>, n) : cudaLaunchKernelEx(&c.c, pass_norm<NORM_MID>, n);
    };
    int expo = 0;
    const int pow2 = frexpf(d.scale, &expo) == 0.5f;
    auto mul = [&](int kind, int l) {
        const Tile& t = pl->tile[kind];
        GemmArgs g = {};
        if (kind == K_LOGITS) {
            g = logits_args(p, t, lrows);
            Config c(dim3(std::min(g.ntiles, p.sms)), 0, st, true);
            c.c.dynamicSmemBytes = block_bytes(p, kind, t, g.ntiles);
            return gemm(EPI_LOGITS, t, c.c, pl->w[kind], pl->a[kind], g);
        }
        g.layer = l; g.D = D; g.rp = p.rp; g.stages = t.stages; g.status = (u32*)d.bar; g.limit = p.wait_ns; g.skip = (const int*)u(p.o.skip);
        g.rows = rows;
        g.kblocks = kind == K_P2 ? kbf : kbd; g.kb_per = (g.kblocks + t.splits - 1) / t.splits;
        g.nfeat = kind == K_QKV ? 3 * D : kind == K_FC ? F : D;
        if (kind == K_QKV) {
            g.bias = f16(d.qkvb, (size_t)l * 3 * D); g.of = (float*)u(p.o.q); g.rowoff = (const long long*)u(p.o.rowoff);
            g.kc = (u16*)d.keys + (size_t)l * d.tmax * D; g.vc = (u16*)d.vals + (size_t)l * d.tmax * D;
            if (many) { g.oh = (u16*)u(p.o.q); g.low = (size_t)d.rows * D; g.a2 = pow2 ? 1.0f / d.scale : 1.0f; }
            if (clear) { g.lens = meta + mt.lens; g.seqs = d.prompts; g.seq_stride = (long long)L * d.tmax * D; g.tmax = d.tmax; }
        } else if (kind == K_FC) {
            g.bias = f16(d.fcb, (size_t)l * F); g.oh = (u16*)u(p.o.gelu); g.pitch = up(F, 64); g.a2 = 2 * d.gelu_a; g.k1 = d.gelu_b * 2.8853900817779268f; g.k2 = d.gelu_c * g.k1;
        } else { g.of = z; g.bias = kind == K_PROJ ? f16(d.ob, (size_t)l * D) : f16(d.pb, (size_t)l * D); }
        g.bn = t.bn; g.ftiles = (g.nfeat + t.bm - 1) / t.bm; g.rtiles = p.rp ? 1 : (g.rows + t.bn - 1) / t.bn; g.ntiles = g.ftiles * g.rtiles * t.splits;
        Config c(dim3(t.bm == 64 ? g.ntiles : t.bm == 256 ? 2 * std::min(g.ntiles, p.sms / 2) : std::min(g.ntiles, p.sms)), 0, st, true, t.bm == 256 ? 2 : 1, true);
        c.c.dynamicSmemBytes = block_bytes(p, kind, t, g.ntiles);
        return gemm(epi_of(kind), t, c.c, pl->w[kind], pl->a[kind], g);
    };
    auto attend = [&](int l) {
        const float* q = (const float*)u(p.o.q);
        const u16 *kc = (const u16*)d.keys + (size_t)l * d.tmax * D, *vc = (const u16*)d.vals + (size_t)l * d.tmax * D;
        const long long ss = (long long)L * d.tmax * D;
        if (many) {
            AttManyArgs a = {(const int4*)(meta + mt.tiles), l, L, D, d.scale, att, (u32*)d.bar, p.wait_ns};
            Config c(dim3(d.H, tiles), AM_THREADS, st, true);
            c.c.dynamicSmemBytes = AM_SMEM;
            return pow2 ? cudaLaunchKernelEx(&c.c, pass_attend_many<true>, p.qmap, p.kmap, p.vmap, a) : cudaLaunchKernelEx(&c.c, pass_attend_many<false>, p.qmap, p.kmap, p.vmap, a);
        }
        AttArgs a = {q, kc, vc, ss, (const int*)d.t, d.t_stride, d.tmax, D, pow2, p.rp, d.scale, att};
        Config c(dim3(d.H, rows, C), shape / 10 * 32, st, true, C);
        c.c.dynamicSmemBytes = (shape / 10) * (shape % 10) * 4096;
        return shape == 83 ? cudaLaunchKernelEx(&c.c, pass_attend<3, 8>, a) : shape == 82 ? cudaLaunchKernelEx(&c.c, pass_attend<2, 8>, a) : shape == 44 ? cudaLaunchKernelEx(&c.c, pass_attend<4, 4>, a) : cudaLaunchKernelEx(&c.c, pass_attend<2, 4>, a);
    };
    TRY(norm(0, 0));
    for (int l = 0; l < L; l++) {
        TRY(mul(K_QKV, l));
        if (l == L - 1 && lrows == 0) break;
        TRY(attend(l));
        TRY(mul(K_PROJ, l));
        TRY(norm(1, l));
        TRY(mul(K_FC, l));
        TRY(mul(K_P2, l));
        TRY(norm(l + 1 < L ? 2 : 3, l));
    }
    if (lrows) TRY(mul(K_LOGITS, 0));
    FinishArgs f = finish(p, lrows);
    if (many) { f.dst = (const int2*)(meta + mt.dst); f.x = (int*)d.x; f.t = (int*)d.t; }
    Config c(dim3(1), 256, st, true);
    TRY(cudaLaunchKernelEx(&c.c, pass_finish, f));
    return 0;
}

// one case per width (units of 256, at most) and warps per row (four, fixed point: two rows; two, fp32: three and four)
#define FEW_EACH(X) X(1, 4, true) X(1, 2, false) X(2, 4, true) X(2, 2, false) X(3, 4, true) X(3, 2, false) X(4, 4, true) X(4, 2, false)
cudaError_t few_launch(cudaLaunchConfig_t& c, int D, bool fixed, const FewQkv& a) {
#define ONE(K, W, F) if (D <= 256 * K && fixed == F) return cudaLaunchKernelEx(&c, few_qkv<K, W, F>, a);
    FEW_EACH(ONE)
#undef ONE
    return cudaErrorInvalidValue;
}
cudaError_t few_launch(cudaLaunchConfig_t& c, int D, bool fixed, const FewMlp& a) {
#define ONE(K, W, F) if (D <= 256 * K && fixed == F) return cudaLaunchKernelEx(&c, few_mlp<K, W, F>, a);
    FEW_EACH(ONE)
#undef ONE
    return cudaErrorInvalidValue;
}
cudaError_t few_launch(cudaLaunchConfig_t& c, bool fixed, const FewAttend& a) {
    return fixed ? cudaLaunchKernelEx(&c, few_attend<true>, a) : cudaLaunchKernelEx(&c, few_attend<false>, a);
}
cudaError_t few_prepare() {
    cudaError_t e = cudaSuccess;
    auto one = [&](auto* f, int bytes = SMEM_MAX - 1024) {
        if (e == cudaSuccess) e = all_shared(f);
        if (e == cudaSuccess) e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
#define ONE(K, W, F) one(few_qkv<K, W, F>); one(few_mlp<K, W, F>);
    FEW_EACH(ONE)
#undef ONE
    one(few_attend<true>, FewAttend::bytes(1024)); one(few_attend<false>, FewAttend::bytes(1024));
    return e;
}

// a step of few sequences
int enqueue_few(Pass& p, cudaStream_t st) {
    const vesta_pass_desc& d = p.d;
    const Few& f = p.few;
    const int D = d.D, F = d.F, R = d.rows;
    const Pass::Plan* pl = nullptr;
    if (int e = plan_for(p, R, R, &pl)) return e;
    auto u = [&](size_t off) { return p.ws + off; };
    auto f16 = [](const void* q, size_t off) { return (const u16*)q + off; };
    const FewPack pk(D, F);
    int expo = 0;
    const int pow2 = frexpf(d.scale, &expo) == 0.5f;
    for (int l = 0; l < d.L; l++) {
        const unsigned char* w = u(p.o.packed) + (size_t)l * pk.layer;
        u16 *kc = (u16*)d.keys + (size_t)l * d.tmax * D, *vc = (u16*)d.vals + (size_t)l * d.tmax * D;
        const long long ss = (long long)d.L * d.tmax * D;
        {
            FewQkv a = {};
            a.n = {D, R, d.eps, u(p.o.after[(l + 1) & 1]), u(p.o.sums[(l + 1) & 1]), f16(d.ln1w, (size_t)l * D), f16(d.ln1b, (size_t)l * D), u(p.o.after[l & 1]), f16(d.ob, (size_t)l * D), u(p.o.sums[l & 1])};
            a.w = w + pk.qkv; a.bias = f16(d.qkvb, (size_t)l * 3 * D); a.tiles = 3 * D / 16; a.per = f.qkv_per; a.q = (float*)u(p.o.q); a.kc = kc; a.vc = vc; a.seq_stride = ss;
            a.x = (const int*)d.x; a.t = (const int*)d.t; a.t_stride = d.t_stride; a.tmax = d.tmax; a.cpos = d.cpos; a.N = d.N; a.first = l == 0; a.wte = (const u16*)d.wte; a.wpe = (const u16*)d.wpe;
            a.pos = (int*)u(p.o.pos); a.skip = (int*)u(p.o.skip); a.bar = (u32*)d.bar;
            Config c(dim3((a.tiles + a.per - 1) / a.per), FEW_THREADS, st, l != 0);
            c.c.dynamicSmemBytes = FewQkv::bytes(D, R, a.per);
            TRY(few_launch(c.c, D, f.fixed, a));
        }
        {
            FewAttend a = {};
            a.a = {(const float*)u(p.o.q), kc, vc, ss, (const int*)d.t, d.t_stride, d.tmax, D, pow2, 0, d.scale, nullptr};
            a.rows = R; a.chunks = f.fixed ? 4 : 2; a.w = w + pk.proj; a.z = u(p.o.after[l & 1]);
            Config c(dim3(FEW_CLUSTER, d.H), FEW_THREADS, st, true, FEW_CLUSTER, true);
            c.c.dynamicSmemBytes = FewAttend::bytes(D);
            TRY(few_launch(c.c, f.fixed, a));
        }
        {
            FewMlp a = {};
            a.n = {D, R, d.eps, u(p.o.after[l & 1]), nullptr, f16(d.ln2w, (size_t)l * D), f16(d.ln2b, (size_t)l * D), u(p.o.sums[l & 1]), f16(d.pb, (size_t)l * D), nullptr};
            a.fc = w + pk.fc; a.p2 = w + pk.p2; a.bias = f16(d.fcb, (size_t)l * F); a.tiles = F / 16; a.per = f.mlp_per;
            a.a2 = 2 * d.gelu_a; a.k1 = d.gelu_b * 2.8853900817779268f; a.k2 = d.gelu_c * a.k1;
            Config c(dim3((a.tiles + a.per - 1) / a.per), FEW_THREADS, st, true);
            // (a block of two tiles has its SM for itself, they are no more than the SMs: two sequences of the small shape, whose 114 KB would
            // fit twice, 170.3 us per step so, 172.2 in pairs)
            c.c.dynamicSmemBytes = std::max(FewMlp::bytes(D, R, a.per), a.per > 1 ? SMEM_MAX / 2 : 0);
            TRY(few_launch(c.c, D, f.fixed, a));
        }
    }
    NormArgs n = {};
    n.D = D; n.rp = p.rp; n.eps = d.eps; n.gain = f16(d.lnfw, 0); n.shift = f16(d.lnfb, 0); n.act = (u16*)u(p.o.fin);
    n.z = (float*)u(p.o.after[(d.L - 1) & 1]); n.more = u(p.o.sums[(d.L - 1) & 1]); n.fixed = f.fixed;
    Config cn(dim3(R), up(D / 4, 32), st, true);
    TRY(cudaLaunchKernelEx(&cn.c, pass_norm<NORM_FINAL>, n));
    const Tile& t = pl->tile[K_LOGITS];
    const GemmArgs g = logits_args(p, t, R);
    Config cg(dim3(std::min(g.ntiles, p.sms)), 0, st, true);
    cg.c.dynamicSmemBytes = block_bytes(p, K_LOGITS, t, g.ntiles);
    TRY(gemm(EPI_LOGITS, t, cg.c, pl->w[K_LOGITS], pl->a[K_LOGITS], g));
    Config cf(dim3(1), 256, st, true);
    TRY(cudaLaunchKernelEx(&cf.c, pass_finish, finish(p, R)));
    return 0;
}
int step(Pass& p, cudaStream_t st) { return p.few.on ? enqueue_few(p, st) : enqueue(p, st, p.d.rows, p.d.logit_rows, 0); }
int pack_few(const Pass& p, cudaStream_t st) {
    const vesta_pass_desc& d = p.d;
    const FewPackArgs a = {d.D, d.F, d.L, (const u16*)d.qkvw, (const u16*)d.ow, (const u16*)d.fcw, (const u16*)d.pw, p.ws + p.o.packed};
    few_pack<<<p.sms * 8, 256, 0, st>>>(a);
    TRY(cudaGetLastError());
    return 0;
}

// No exception leaves an entry of the library.
template <class F> int guarded(F f) {
    try { return f(); }
    catch (const std::exception& e) { return fail(-1, e.what()); }
}

// a decode step as a graph, captured on a stream of its own, in place of the one that the pass has
int capture(Pass* p) {
    cudaStream_t st = nullptr;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    int e = 0;
    cudaError_t ce = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (ce == cudaSuccess) ce = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (ce == cudaSuccess) {
        e = guarded([&] { return step(*p, st); });      // (the capture ends whatever happens in it)
        ce = cudaStreamEndCapture(st, &g);
    }
    if (ce == cudaSuccess && !e) ce = cudaGraphInstantiate(&ge, g, 0);
    if (ge) {
        if (p->graph) cudaGraphExecDestroy(p->graph);
        p->graph = ge;
    }
    if (g) cudaGraphDestroy(g);
    if (st) cudaStreamDestroy(st);
    return ce != cudaSuccess && !e ? cuda_fail(ce, "vesta_pass: graph of a step") : e;
}

// sizes, tensor maps and, for decode steps, the graph of a pass
int make(Pass* p, const vesta_pass_desc* d, unsigned char* workspace, bool graph) {
    int e = plan(*p, d);
    if (!e) e = check(*d);
    if (!e && (size_t)workspace % 256) e = fail(-1, "vesta_pass: the workspace starts on a 256-byte boundary");
    p->ws = workspace;
    if (!e) { cudaError_t ce = p->few.on ? few_prepare() : cudaSuccess; if (ce == cudaSuccess) ce = prepare_all(); if (ce != cudaSuccess) e = cuda_fail(ce, "cudaFuncSetAttribute"); }
    if (!e && d->prompts) {
        const unsigned long long D = d->D, planes = (unsigned long long)d->prompts * d->L;
        e = vesta_rt::tensor_map(&p->kmap, d->keys, D, d->tmax, planes, D * 2, D * 2 * d->tmax, 128, 1);
        if (!e) e = vesta_rt::tensor_map(&p->qmap, p->ws + p->o.q, D, d->rows, 2, D * 2, D * 2 * d->rows, 128, 1);
        if (!e) e = vesta_rt::tensor_map(&p->vmap, d->vals, D, d->tmax, planes, D * 2, D * 2 * d->tmax, 128, 1);
    }
    if (!e && graph) e = capture(p);
    return e;
}

// whole prompts: the passes of a call, their metadata and the status word
int read_prompts(Pass* p, cudaStream_t st, const int* tokens, int ld, const int* lens, unsigned* status) {
    const vesta_pass_desc& d = p->d;
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
    std::vector<int> written(B);
    int s = 0, pos = 0;                          // next position to read
    for (int c = 0; c < passes; c++) {
        int* m = p->host + (size_t)c * mt.words;
        int n = 0, lrows = 0;
        runs.clear();
        while (n < per && s < B) {
            const int take = std::min(per - n, lens[s] - pos);
            for (int i = 0; i < take; i++) { m[mt.x + n + i] = tokens[(size_t)s * ld + pos + i]; m[mt.t + n + i] = pos + i; m[mt.seq + n + i] = s; }
            for (int i = 0; i < take; i += 128) runs.push_back(Run{n + i, std::min(128, take - i), s, pos + i});
            n += take; pos += take;
            if (pos == lens[s]) {
                m[mt.want + lrows] = n - 1; m[mt.dst + 2 * lrows] = s; m[mt.dst + 2 * lrows + 1] = lens[s];
                lrows++; s++; pos = 0;
            }
        }
        // the runs that see most positions first
        std::stable_sort(runs.begin(), runs.end(), [](const Run& a, const Run& b) { return a.pos + a.rows > b.pos + b.rows; });
        for (size_t i = 0; i < runs.size(); i++) { int* t = m + mt.tiles + 4 * i; t[0] = runs[i].first; t[1] = runs[i].rows; t[2] = runs[i].seq; t[3] = runs[i].pos; }
        // rows written by the first pass: everything behind them is cleared there, what later passes will write included
        if (c == 0) for (int i = 0; i < B; i++) written[i] = i < s ? lens[i] : i == s ? pos : 0;
        for (int i = 0; i < B; i++) m[mt.lens + i] = written[i];
        TRY(cudaMemcpyAsync(p->ws + p->o.meta, m, (size_t)mt.words * 4, cudaMemcpyHostToDevice, st));
        if (int e = enqueue(*p, st, n, lrows, (int)runs.size(), c == 0)) return e;
    }
    unsigned* word = (unsigned*)(p->host + words - 4);
    TRY(cudaMemcpyAsync(word, d.bar, 4, cudaMemcpyDeviceToHost, st));
    TRY(cudaStreamSynchronize(st));
    *status = *word;
    return 0;
}

}  // namespace

namespace vesta_rt {
namespace {
// the device of a pass for the calls of a scope (launches go to a stream of the current device)
struct OnDevice {
    int was = 0, dev;
    explicit OnDevice(int d) : dev(d) { if (cudaGetDevice(&was) == cudaSuccess && was != dev) cudaSetDevice(dev); }
    ~OnDevice() { if (was != dev) cudaSetDevice(was); }
};
}
int pass_steps(void* pass, void* stream, int steps) {
    Pass* p = (Pass*)pass;
    const OnDevice on(p->dev);
    cudaStream_t st = (cudaStream_t)stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TRY(cudaStreamIsCapturing(st, &cap));
    return guarded([&]() -> int {
        for (int i = 0; i < steps; i++) {
            if (cap != cudaStreamCaptureStatusNone || !p->graph) { if (int e = step(*p, st)) return e; }
            else TRY(cudaGraphLaunch(p->graph, st));
        }
        return 0;
    });
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

int vesta_pass_tiles(const vesta_pass_desc* d, int rows, int logit_rows, int* out) {
    Pass p{};
    if (!out || !d || rows < 1 || rows > d->rows || logit_rows < 0 || logit_rows > d->logit_rows) return fail(-1, "vesta_pass_tiles: bad argument");
    if (int e = plan(p, d)) return e;
    for (int k = 0; k < 5; k++) {
        const Tile t = tile_of(p, k, rows, logit_rows);
        const int feat = k == K_QKV ? 3 * d->D : k == K_FC ? d->F : k == K_LOGITS ? d->N : d->D, n = k == K_LOGITS ? std::max(logit_rows, 1) : rows;
        const int ntiles = (feat + t.bm - 1) / t.bm * (p.rp ? 1 : (n + t.bn - 1) / t.bn) * t.splits;
        const int v[5] = {t.bm, t.bn, t.stages, t.splits, (int)block_bytes(p, k, t, ntiles)};
        std::copy(v, v + 5, out + 5 * k);
    }
    return 0;
}

int vesta_pass_create(const vesta_pass_desc* d, void* workspace, int graph, void** out) {
    if (!out || !workspace) return fail(-1, "vesta_pass_create: null argument");
    Pass* p = nullptr;
    if (const int e = guarded([&] { p = new Pass{}; return make(p, d, (unsigned char*)workspace, graph != 0); })) { vesta_pass_release(p); return e; }
    *out = p;
    return 0;
}

int vesta_pass_prompts(void* pass, void* stream, const int* tokens, int ld, const int* lens, unsigned* status) {
    Pass* p = (Pass*)pass;
    if (!p || !p->d.prompts || !tokens || !lens || !status) return fail(-1, "vesta_pass_prompts: bad argument");
    const int e = guarded([&] { return read_prompts(p, (cudaStream_t)stream, tokens, ld, lens, status); });
    if (e) cudaStreamSynchronize((cudaStream_t)stream);                  // (the next call writes the pinned metadata that copies may still read)
    return e;
}

int vesta_pass_pack(void* pass, void* stream) {
    Pass* p = (Pass*)pass;
    if (!p) return fail(-1, "vesta_pass_pack: null argument");
    if (!p->few.on) return 0;
    const vesta_rt::OnDevice on(p->dev);
    return pack_few(*p, (cudaStream_t)stream);
}

int vesta_pass_wait_limit(void* pass, unsigned long long ns) {
    Pass* p = (Pass*)pass;
    if (!p) return fail(-1, "vesta_pass_wait_limit: null argument");
    const vesta_rt::OnDevice on(p->dev);
    p->wait_ns = ns ? ns : WAIT_NS;
    return p->graph ? capture(p) : 0;
}

void vesta_pass_release(void* pass) {
    Pass* p = (Pass*)pass;
    if (!p) return;
    if (p->graph) cudaGraphExecDestroy(p->graph);
    if (p->host) cudaFreeHost(p->host);
    delete p;
}

}  // extern "C"
