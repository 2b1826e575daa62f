// Kernels of one forward pass over a set of rows, written for sm_100a: the rows are the sequences of a decode step or the
// (sequence, position) pairs of prompts. A pass is a chain of small kernels per layer,
//
//     norm | QKV | attention | projection | norm | FC | MLP projection
//
// launched with programmatic stream serialization: a kernel starts while its predecessor runs, does what does not depend
// on it (barriers, tensor memory, its weights into shared memory) and waits (griddepcontrol.wait) before it touches what
// the predecessor writes. Measured on B200 in a CUDA graph: 1.15 to 1.25 us per kernel of such a chain, a load from L2
// and a store included (148 blocks; 1.4 without the early start, 2.4 us and more for a barrier across one persistent
// kernel), and the weights of several kernels ahead stream in meanwhile, as far as shared memory goes.
//
// Contractions (pass_gemm) run on tcgen05.mma with the output features as the rows of the product (operand A: the
// weights as they are stored, [fold][feature], i.e. M-major; the table of the logits K-major) and the rows of the pass as
// its columns (operand B, fp16 [row][fold]). So few rows cost few columns, and a weight element is read by one block (per tile of rows).
// Rows whose activations are multiplied at fp32 accuracy (`rp` > 0) pass as two planes, fp16 head and fp16 remainder,
// in the columns [0, rp) and [rp, 2 rp) of the same product.
// The projections add into the residual stream with reductions. A fold that is one block's adds once per element: the same bits
// every time. A fold that is cut over blocks adds its parts in the order in which the blocks finish: the last bits of a pass may
// differ from run to run (stored apart and added in order by the norm behind they were equal, and 2 to 6 % slower).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace vesta_pass {

typedef unsigned int u32;
typedef unsigned long long u64;
typedef unsigned short u16;

// ---- small wrappers -------------------------------------------------------------------------------------------------
__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ u64 now_ns() { u64 t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
__device__ __forceinline__ u32 pack_h2(float lo, float hi) { u32 r; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo)); return r; }
__device__ __forceinline__ float h_lo(u32 w) { float f; asm("{.reg .b16 l,h; mov.b32 {l,h}, %1; cvt.f32.f16 %0, l;}" : "=f"(f) : "r"(w)); return f; }
__device__ __forceinline__ float h_hi(u32 w) { float f; asm("{.reg .b16 l,h; mov.b32 {l,h}, %1; cvt.f32.f16 %0, h;}" : "=f"(f) : "r"(w)); return f; }
__device__ __forceinline__ float h2f(u16 h) { float f; asm("cvt.f32.f16 %0, %1;" : "=f"(f) : "h"(h)); return f; }
__device__ __forceinline__ u16 f2h(float f) { u16 h; asm("cvt.rn.f16.f32 %0, %1;" : "=h"(h) : "f"(f)); return h; }
__device__ __forceinline__ float fast_exp(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f)); return y; }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(u32 bar, u32 count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void mbar_expect(u32 bar, u32 bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ bool mbar_try(u32 bar, u32 parity) {
    u32 ok;
    asm volatile("{.reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tma3(u32 dst, const CUtensorMap* m, int x, int y, int z, u32 bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(dst), "l"(m), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// the same into this block of a pair, counted on a barrier of the pair's first block (no multicast)
__device__ __forceinline__ void tma3_pair(u32 dst, const CUtensorMap* m, int x, int y, int z, u32 bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 :: "r"(dst), "l"(m), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// a shared-memory address of this block as the same address of block `rank` of its cluster
__device__ __forceinline__ u32 of_block(u32 a, u32 rank) {
    u32 r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ u32 of_first(u32 a) { return of_block(a, 0); }
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// arrives on `bar` (of a pair: at that address in both blocks) when the products issued so far are done
template <bool PAIR> __device__ __forceinline__ void tc_commit(u32 bar) {
    if (PAIR) asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" :: "r"(bar), "h"((u16)3) : "memory");
    else asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ u32 elect_one() {
    u32 leader;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leader));
    return leader;
}

// The residual stream: fp32, or 64-bit fixed point (36 fractional bits: finer than fp32 below 2^27) whose integer additions give the
// same bits in every order.
#define STATE_SCALE 68719476736.0f
template <bool FIXED> struct State;
template <> struct State<false> {
    static __device__ __forceinline__ float4 load(const void* z, size_t i) { return __ldcg(reinterpret_cast<const float4*>((const float*)z + i)); }
    static __device__ __forceinline__ float4 load(const void* z, const void* more, size_t i) {       // the sum of two vectors
        const float4 a = load(z, i), b = load(more, i);
        return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
    static __device__ __forceinline__ void store(void* z, size_t i, float4 v) { *reinterpret_cast<float4*>((float*)z + i) = v; }
    static __device__ __forceinline__ void add1(void* z, size_t i, float v) { asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" :: "l"((float*)z + i), "f"(v) : "memory"); }
    static __device__ __forceinline__ void add(void* z, size_t i, float4 v) {
        asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1,%2,%3,%4};" :: "l"((float*)z + i), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    }
};
template <> struct State<true> {
    static __device__ __forceinline__ float from(long long v) { return __ll2float_rn(v) * (1.0f / STATE_SCALE); }
    static __device__ __forceinline__ float4 load(const void* z, size_t i) {
        const longlong2* p = reinterpret_cast<const longlong2*>((const long long*)z + i);
        const longlong2 a = __ldcg(p), b = __ldcg(p + 1);
        return make_float4(from(a.x), from(a.y), from(b.x), from(b.y));
    }
    static __device__ __forceinline__ float4 load(const void* z, const void* more, size_t i) {
        const longlong2 *p = reinterpret_cast<const longlong2*>((const long long*)z + i), *q = reinterpret_cast<const longlong2*>((const long long*)more + i);
        const longlong2 a = __ldcg(p), b = __ldcg(p + 1), c = __ldcg(q), d = __ldcg(q + 1);
        return make_float4(from(a.x + c.x), from(a.y + c.y), from(b.x + d.x), from(b.y + d.y));
    }
    static __device__ __forceinline__ void store(void* z, size_t i, float4 v) {
        longlong2* p = reinterpret_cast<longlong2*>((long long*)z + i);
        p[0] = make_longlong2(__float2ll_rn(v.x * STATE_SCALE), __float2ll_rn(v.y * STATE_SCALE));
        p[1] = make_longlong2(__float2ll_rn(v.z * STATE_SCALE), __float2ll_rn(v.w * STATE_SCALE));
    }
    static __device__ __forceinline__ void add1(void* z, size_t i, float v) {
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" :: "l"((long long*)z + i), "l"(__float2ll_rn(v * STATE_SCALE)) : "memory");
    }
    static __device__ __forceinline__ void add(void* z, size_t i, float4 v) { add1(z, i, v.x); add1(z, i + 1, v.y); add1(z, i + 2, v.z); add1(z, i + 3, v.w); }
};

// Every wait gives up after `limit` nanoseconds (half a second): it leaves a code in the status word, a flag that ends the other
// waits of the block (of the pair: `peer` is the flag of the other block) and the abort flag: this pass publishes no token or
// position, and every later one is refused. The block runs to its end: a warp whose wait gave up goes on through the
// barriers that other warps of the block wait at, and does nothing between them.
struct Wait { u32 dead, peer; u32* status; u64 limit; };
// (All by value, and the limit a parameter of the kernel: a structure passed by reference gave every kernel a stack frame, and a
// limit read from memory here held up the next try: together 0.2 to 0.6 us per contraction, 16 sequences of the XL shape
// 5,064 -> 5,257 us per four steps, 8 x 128 prompts 576 -> 600.)
__device__ __noinline__ bool mbar_wait_slow(u32 bar, u32 parity, u32 code, u32 dead, u32 peer, u32* status, u64 limit) {
    const u64 t0 = now_ns();
    while (!mbar_try(bar, parity)) {                     // (a try holds the thread for up to 4 us)
        u32 over;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(over) : "r"(dead) : "memory");
        if (over) return false;
        if (now_ns() - t0 > limit) {
            atomicCAS(status, 0u, code | (blockIdx.x << 16));
            atomicExch(status + 2, 1u);
            asm volatile("st.volatile.shared.u32 [%0], %1;" :: "r"(dead), "r"(1u) : "memory");
            if (peer) asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(peer), "r"(1u) : "memory");
            return false;
        }
    }
    return true;
}
// After a wait that gave up: copies and products in flight land (in a few microseconds) before the block's shared memory and
// tensor memory go to another.
__device__ __noinline__ void settle() {
    const u64 t0 = now_ns();
    while (now_ns() - t0 < 2000000ull) { }
}
__device__ __forceinline__ bool mbar_wait(u32 bar, u32 parity, const Wait& w, u32 code) { return mbar_try(bar, parity) || mbar_wait_slow(bar, parity, code, w.dead, w.peer, w.status, w.limit); }

// ---- contractions ---------------------------------------------------------------------------------------------------
enum { EPI_QKV = 0, EPI_ADD = 1, EPI_GELU = 2, EPI_LOGITS = 3 };

struct GemmArgs {
    int layer, nfeat, kblocks, kb_per, rows, rp, stages;
    int bn, ftiles, rtiles, ntiles;  // rows per tile (a multiple of 16); tiles of features, of rows, in all (with the parts of the fold)
    int D, pitch;                    // GELU: elements from a row to the next, nfeat rounded up to 64: the padding stays zero
    const u16* bias;                 // of the layer
    float* of;                       // QKV: queries [row][D] (prompts: `oh`); ADD: vector added to [row][nfeat]; LOGITS: logits [row][nfeat]
    size_t low;                      // QKV, prompts: from a query's heads to its remainders
    u16* oh;                         // GELU: [row][pitch], the remainder plane rp rows further; QKV, prompts: queries times a2, [fp16 head, remainder][row][D]
    u16 *kc, *vc;                    // QKV: the caches at this layer
    const long long* rowoff;         // QKV: element offset of every row's position in the caches (-1: none)
    const int* skip;                 // not zero: the pass was refused, nothing may be written that outlives it
    u64* best;                       // LOGITS: packed (value, ~index) maximum of every row
    u32* status;
    u64 limit;                       // of a wait, ns
    float a2, k1, k2;                // GELU: see gelu_tanh; QKV, prompts: a2 = 1 / scale where that is a power of two
    // QKV, prompts: one more warp zeroes this layer's cache rows behind the first lens[sequence], which this pass writes
    const int* lens;
    long long seq_stride;
    int seqs, tmax;
};

// shared-memory operand descriptors, 128-byte swizzle. K-major: rows of 128 bytes (64 fold indices), groups of eight rows
// 1024 bytes apart. M-major: rows of 128 bytes hold 64 features of one fold index, groups of eight fold indices 1024
// bytes apart, the next 64 features `chunk` bytes further (one box).
__device__ __forceinline__ u64 desc_k(u32 a) { return (u64)((a & 0x3FFFFu) >> 4) | ((u64)1 << 16) | ((u64)(1024 >> 4) << 32) | ((u64)1 << 46) | ((u64)2 << 61); }
__device__ __forceinline__ u64 desc_m(u32 a, u32 chunk) { return (u64)((a & 0x3FFFFu) >> 4) | ((u64)(chunk >> 4) << 16) | ((u64)(1024 >> 4) << 32) | ((u64)1 << 46) | ((u64)2 << 61); }

template <int N> struct Int { static constexpr int n = N; };
// CH consecutive columns of this thread's tensor-memory lane
__device__ __forceinline__ void tm_ld(float (&r)[16], u32 addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]),
                   "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tm_ld(float (&r)[8], u32 addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tm_ld(float (&r)[4], u32 addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(addr) : "memory");
}
// the loads have arrived: the values pass through here, so that nothing that uses them is moved in front of the wait
__device__ __forceinline__ void tm_wait(float (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]), "+f"(r[8]), "+f"(r[9]), "+f"(r[10]),
                 "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15]) :: "memory");
}
__device__ __forceinline__ void tm_wait(float (&r)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]) :: "memory");
}
__device__ __forceinline__ void tm_wait(float (&r)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]) :: "memory");
}
// tanh-GELU: a v (1 + tanh(b (v + c v^3))) with tanh(u) = 1 - 2 / (1 + e^(2u)): 2a v (1 - 1 / (1 + 2^(v (k1 + k2 v^2)))),
// k1 = 2 b log2(e), k2 = c k1
__device__ __forceinline__ float gelu_tanh(float v, float a2, float k1, float k2) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v * fmaf(v * v, k2, k1)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    const float w = a2 * v;
    return fmaf(-w, r, w);
}
// orderable key of (value, index): larger value wins, then the lower index
__device__ __forceinline__ u64 best_key(int ordered, u32 n) { return ((u64)((u32)ordered ^ 0x80000000u) << 32) | (u64)(0xFFFFFFFFu - n); }

// Shared memory of a block: the stages, then full and empty barriers, the accumulators' full and empty barriers, the
// tensor-memory address and the dead flag; per accumulator the row offsets (QKV) or the warps' best keys (LOGITS).
template <int BM> struct GemmShape {
    static constexpr bool PAIR = BM == 256;              // two blocks of a cluster share the tile
    static constexpr int AM = PAIR ? 128 : BM;           // features per block
    static constexpr int KS = BM == 64 ? 4 : 1;          // blocks of 64 fold indices per stage
    static constexpr int EW = 8;                         // warps that read the accumulators: two per quarter of the lanes
    static constexpr int THREADS = 64 + 32 * EW;
    static __host__ __device__ constexpr int box(int bn) { return PAIR ? bn / 2 : bn; }       // rows per block
    static __host__ __device__ constexpr int stage(int bn) { return KS * (AM + box(bn)) * 128; }
    static __host__ __device__ constexpr int tail(int stages, int bn) { return 2 * stages * 8 + 48 + bn * 8 * 4; }
    static __host__ __device__ constexpr int bytes(int stages, int bn) { return stages * stage(bn) + tail(stages, bn) + 1024; }
    static __host__ __device__ constexpr int columns(int bn, bool two) { int c = 32; while (c < (two ? 2 * bn : bn)) c *= 2; return c; }
};
__device__ __forceinline__ void st_u16(u16* p, u16 v, bool yes) {
    asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p st.global.u16 [%0], %1;}" :: "l"(p), "h"(v), "r"((int)yes) : "memory");
}
__device__ __forceinline__ void st_f32(float* p, float v, bool yes) {
    asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p st.global.f32 [%0], %1;}" :: "l"(p), "f"(v), "r"((int)yes) : "memory");
}

__device__ __forceinline__ void add_f32(float* p, float v, bool yes) {
    asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; @p red.relaxed.gpu.global.add.f32 [%0], %1;}" :: "l"(p), "f"(v), "r"((int)yes) : "memory");
}

// Tiles of BM features x bn rows over kb_per blocks of 64 fold indices; a block takes the tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... Warp 0 loads (one lane), warp 1 issues the products, the others read the accumulators; with
// more tiles than blocks two accumulators alternate, so that a tile's epilogue runs under the next one's products.
//   BM = 64: few rows, one tile per block. What counts is the chain wait - operand - products - epilogue: the block's
//     whole share of the weights is in flight before it waits for its predecessor, four blocks of the fold per stage (a
//     stage costs the issuing warps 0.1 us whatever its size: 12 blocks of 64 x 16 took 2.0 us one by one, 1.0 in fours).
//   BM = 128: many rows. What bounds it is the path from L2 into the SMs, 120 GB/s each whatever the tile: 128 x 192 tiles
//     1,160 to 1,200 TFLOP/s.
//   BM = 256: many rows, two blocks of a cluster with one product of 256 rows (cta_group::2): each loads its own 128 features and
//     half the rows of the tile, so that a 256 x 256 tile costs an SM 32 KB per block of the fold instead of 48.
#define CLEAR_ROWS 16
template <int BM, int EPI>
__global__ void __launch_bounds__(GemmShape<BM>::THREADS + (EPI == EPI_QKV ? 32 : 0)) pass_gemm(const __grid_constant__ CUtensorMap wm, const __grid_constant__ CUtensorMap am, const __grid_constant__ GemmArgs g) {
    using S = GemmShape<BM>;
    constexpr int KS = S::KS, EW = S::EW, AM = S::AM;
    constexpr bool PAIR = S::PAIR;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int st = g.stages, bn = g.bn, stage = S::stage(bn);
    const u32 sbase = smem_u32(smem), bars = sbase + st * stage, tmf = bars + 2 * st * 8, tme = tmf + 16;
    unsigned char* tail = smem + st * stage + 2 * st * 8 + 32;
    volatile int* dead = reinterpret_cast<volatile int*>(tail + 4);
    volatile u32* tmem_p = reinterpret_cast<volatile u32*>(tail);
    u64* side = reinterpret_cast<u64*>(tail + 16);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)(blockIdx.x & 1) : 0;                             // block of the pair; the first one issues the products
    const int t_first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, t_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const bool two = g.ntiles > t_step;
    const int cols = S::columns(bn, two);
    const Wait w{smem_u32(tail + 4), PAIR ? of_block(smem_u32(tail + 4), rank ^ 1) : 0u, g.status, g.limit};
    if (threadIdx.x == 0) {
        *dead = 0;
        for (int i = 0; i < st; i++) { mbar_init(bars + i * 8, 1); mbar_init(bars + (st + i) * 8, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(tmf + i * 8, 1); mbar_init(tme + i * 8, PAIR ? 2 * EW : EW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&am) : "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tail)), "r"(cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tail)), "r"(cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (PAIR) cluster_sync();                                                      // the other block's barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x == 0) dep_launch();              // (after the allocation: the blocks of the next kernel queue behind it)
    const u32 tmem = *tmem_p;
    const int per = g.ftiles * g.rtiles;

    if (warp == 0) {
        if (elect_one()) {
            int s = 0, ph = 1;
            bool first = true;
            for (int t = t_first; t < g.ntiles; t += t_step) {
                const int z = t / per, r = t - z * per, rt = r / g.ftiles, f0 = (r - rt * g.ftiles) * BM + rank * AM, row0 = rt * bn + rank * S::box(bn);
                const int kb0 = z * g.kb_per, nst = (min(g.kb_per, g.kblocks - kb0) + KS - 1) / KS;
                auto load = [&](u32 dst, const CUtensorMap* m, int x, int y, int zz, u32 bar) {
                    if (PAIR) tma3_pair(dst, m, x, y, zz, bar); else tma3(dst, m, x, y, zz, bar);
                };
                auto load_w = [&](int slot, int i) {
                    const u32 dst = sbase + slot * stage, bar = PAIR ? of_first(bars + slot * 8) : bars + slot * 8;
                    if (!PAIR || rank == 0) mbar_expect(bars + slot * 8, PAIR ? 2 * stage : stage);
                    if (EPI == EPI_LOGITS) load(dst, &wm, 0, f0, kb0 + i * KS, bar);
                    else {
                        load(dst, &wm, f0, (kb0 + i * KS) * 64, g.layer, bar);
                        if (AM == 128) load(dst + KS * 8192, &wm, f0 + 64, (kb0 + i * KS) * 64, g.layer, bar);
                    }
                };
                auto load_a = [&](int slot, int i) {
                    load(sbase + slot * stage + KS * AM * 128, &am, 0, row0, kb0 + i * KS, PAIR ? of_first(bars + slot * 8) : bars + slot * 8);
                };
                int i = 0;
                if (first) {
                    // the weights do not depend on the predecessor
                    const int pre = min(st, nst);
                    for (; i < pre; i++) load_w(i, i);
                    dep_wait();
                    for (i = 0; i < pre; i++) load_a(i, i);
                    s = pre; if (s == st) { s = 0; ph = 0; }
                    first = false;
                }
                for (; i < nst; i++) {
                    if (!mbar_wait(bars + (st + s) * 8, ph, w, 0xB00u)) break;
                    load_w(s, i);
                    load_a(s, i);
                    if (++s == st) { s = 0; ph ^= 1; }
                }
                if (*dead) break;
            }
        }
    } else if (warp == 1) {
        // fp32 accumulators, fp16 operands; A M-major (bit 15) except for the table of the logits
        const u32 idesc = (1u << 4) | (EPI == EPI_LOGITS ? 0u : (1u << 15)) | ((u32)(bn >> 3) << 17) | ((u32)(BM >> 4) << 24);
        constexpr int AKB = EPI == EPI_LOGITS ? AM * 128 : 8192, AK = EPI == EPI_LOGITS ? 32 : 2048;   // bytes to the next block, to the next 16 fold indices
        int s = 0, ph = 0, n = 0;
        bool ok = !PAIR || rank == 0;
        for (int t = t_first; t < g.ntiles && ok; t += t_step, n++) {
            const int kb0 = (t / per) * g.kb_per, nkb = min(g.kb_per, g.kblocks - kb0), nst = (nkb + KS - 1) / KS, b = n & 1;
            if (n >= 2) ok = !__any_sync(0xffffffffu, !mbar_wait(tme + b * 8, ((n >> 1) & 1) ^ 1, w, 0xB30u));
            const u32 acc = tmem + (b ? bn : 0);
            for (int i = 0; i < nst && ok; i++) {
                ok = !__any_sync(0xffffffffu, !mbar_wait(bars + s * 8, ph, w, 0xB10u));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // (the elected lane is asked for here, next to the products: under a predicate that comes from further away a
                // product costs 90 cycles instead of the 20 to 40 its operands take: the descriptors then pass to uniform
                // registers one by one)
                if (elect_one()) {
                    const u32 a = sbase + s * stage;
                    const u64 ad = EPI == EPI_LOGITS ? desc_k(a) : desc_m(a, KS * 8192), bd = desc_k(a + KS * AM * 128);
#pragma unroll
                    for (int kb = 0; kb < KS; kb++)
                        if (KS == 1 || i * KS + kb < nkb) {
                            const u64 bk = bd + (u64)((kb * bn * 128) >> 4);
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                if (PAIR)
                                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                                 :: "r"(acc), "l"(ad + (kb * AKB + k * AK) / 16), "l"(bk + 2 * k), "r"(idesc), "r"((i | kb | k) ? 1u : 0u) : "memory");
                                else
                                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                                 :: "r"(acc), "l"(ad + (kb * AKB + k * AK) / 16), "l"(bk + 2 * k), "r"(idesc), "r"((i | kb | k) ? 1u : 0u) : "memory");
                            }
                        }
                    tc_commit<PAIR>(bars + (st + s) * 8);
                    if (i == nst - 1) tc_commit<PAIR>(tmf + b * 8);
                }
                __syncwarp();
                if (++s == st) { s = 0; ph ^= 1; }
            }
        }
    } else if (EPI == EPI_QKV && warp == EW + 2) {
        // Nothing waits for these rows before the attention and they wait for nothing: they leave in the shadow of the
        // products, which need little of the memory. (As a kernel of its own on another stream the clearing delayed the chain:
        // none of its kernels started early until it was done; as blocks of the attention it was that kernel's tail.)
        const int per_row = g.D / 8, parts = (g.tmax + CLEAR_ROWS - 1) / CLEAR_ROWS;
        for (int j = blockIdx.x; j < 2 * g.seqs * parts; j += gridDim.x) {
            const int sq = j / (2 * parts), r = j - sq * 2 * parts, part = r >> 1;
            const int lo = max(part * CLEAR_ROWS, __ldg(g.lens + sq)) * per_row, hi = min((part + 1) * CLEAR_ROWS, g.tmax) * per_row;
            uint4* p = reinterpret_cast<uint4*>(((r & 1) ? g.vc : g.kc) + sq * g.seq_stride);
            for (int i = lo + lane; i < hi; i += 32) p[i] = make_uint4(0, 0, 0, 0);
        }
    } else {
        const int quarter = warp & 3, ew = warp - 2, et = threadIdx.x - 64;
        const int fl = AM == 128 ? quarter * 32 + lane : quarter * 16 + lane;      // (a product of 64 rows leaves row m in lane 32 (m / 16) + m % 16)
        bool waited = false, skip = false, ok = true;
        int n = 0;
        u64 off = ~0ull;                                                           // QKV: a row's offset in the caches, one tile ahead
        auto row_offset = [&](int t) {
            const int i = (t - t / per * per) / g.ftiles * bn + et;
            return t < g.ntiles && et < bn && i < g.rows && !skip ? (u64)__ldcg(g.rowoff + i) : ~0ull;
        };
        for (int t = t_first; t < g.ntiles; t += t_step, n++) {
            const int z = t / per, r0 = t - z * per, rt = r0 / g.ftiles, f0 = (r0 - rt * g.ftiles) * BM + rank * AM, row0 = rt * bn, b = n & 1;
            const int f = f0 + fl;
            const bool own = (AM == 128 || lane < 16) && f < g.nfeat;
            float bias = 0.f;
            if ((EPI == EPI_QKV || EPI == EPI_GELU || (EPI == EPI_ADD && z == 0)) && own) bias = h2f(__ldg(g.bias + f));
            if (!waited) {
                dep_wait();
                waited = true;
                skip = (EPI == EPI_QKV || EPI == EPI_LOGITS) ? __ldcg(g.skip) != 0 : false;
                if (EPI == EPI_QKV) off = row_offset(t);
            }
            const int live = min(g.rp ? g.rp : bn, g.rows - row0);                 // rows of this tile
            if (EPI == EPI_QKV) {
                // (everyone is past the previous tile's offsets but one: two buffers)
                if (et < bn) side[b * bn + et] = off;
                off = row_offset(t + t_step);
                asm volatile("bar.sync 1, %0;" :: "n"(EW * 32) : "memory");
            }
            // the warps of a quarter share the rows
            const int share = live > EW ? (live + 2 * EW - 1) / (2 * EW) * 8 : 4;
            const int c_lo = (ew >> 2) * share, c_hi = min(live, c_lo + share);
            if (ok) ok = !__any_sync(0xffffffffu, !mbar_wait(tmf + b * 8, (n >> 1) & 1, w, 0xB20u));
            if (!ok) {                                                             // (another warp may have seen the same tile complete: it waits at these)
                if (EPI == EPI_LOGITS) {
                    asm volatile("bar.sync 1, %0;" :: "n"(EW * 32) : "memory");
                    if (two) asm volatile("bar.sync 1, %0;" :: "n"(EW * 32) : "memory");
                }
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const u32 ta = tmem + ((u32)(quarter * 32) << 16) + (b ? bn : 0);
            const int part = EPI == EPI_QKV ? f / g.D : 0;                         // 0 query, 1 key, 2 value (a warp never straddles two)
            u16* cache = EPI == EPI_QKV ? (part == 1 ? g.kc : g.vc) + (f - part * g.D) : (u16*)0;
            // CH rows at a time (no branch per row: their chains of arithmetic overlap, only the stores are predicated); the last
            // four or fewer on their own
            auto rows_of = [&](auto CHC, int c0) {
                constexpr int CH = decltype(CHC)::n;
                int m = min(CH, c_hi - c0);
                float v[CH];
                tm_ld(v, ta + c0);
                if (BM == 64 && g.rp) {
                    float q[CH];
                    tm_ld(q, ta + g.rp + c0);
                    tm_wait(v);
                    tm_wait(q);
#pragma unroll
                    for (int i = 0; i < CH; i++) v[i] += q[i];
                } else tm_wait(v);
                const int row = row0 + c0;
#pragma unroll
                for (int i = 0; i < CH; i++) {
                    v[i] += bias;
                    if (EPI == EPI_GELU) v[i] = gelu_tanh(v[i], g.a2, g.k1, g.k2);
                }
                if (!own) m = 0;
                if (EPI == EPI_QKV) {
                    if (part == 0 && g.oh) {
                        u16* dst = g.oh + (size_t)row * g.D + f;
#pragma unroll
                        for (int i = 0; i < CH; i += 2, dst += 2 * g.D) {
                            const float a = v[i] * g.a2, c = v[i + 1] * g.a2;
                            const u32 h = pack_h2(a, c), r = pack_h2(a - h_lo(h), c - h_hi(h));
                            st_u16(dst, (u16)h, i < m); st_u16(dst + g.D, (u16)(h >> 16), i + 1 < m);
                            st_u16(dst + g.low, (u16)r, i < m); st_u16(dst + g.low + g.D, (u16)(r >> 16), i + 1 < m);
                        }
                    } else if (part == 0) {
                        float* dst = g.of + (size_t)row * g.D + f;
#pragma unroll
                        for (int i = 0; i < CH; i++, dst += g.D) st_f32(dst, v[i], i < m);
                    } else {
#pragma unroll
                        for (int i = 0; i < CH; i += 2) {
                            const longlong2 o = *reinterpret_cast<const longlong2*>(side + b * bn + c0 + i);
                            const u32 h = pack_h2(v[i], v[i + 1]);                 // (one conversion for two: alone each runs at a quarter of the rate)
                            st_u16(cache + o.x, (u16)h, i < m && o.x >= 0);
                            st_u16(cache + o.y, (u16)(h >> 16), i + 1 < m && o.y >= 0);
                        }
                    }
                } else if (EPI == EPI_ADD) {
                    // (Reading, adding and storing waited for L2 chunk by chunk: 15 us at 9,216 rows x 768 x 768. Parts of a cut fold
                    // add here too: stored one by one and added by the norm behind they cost every pass more, 256 sequences
                    // 801 -> 762 us per step, 16 of the XL shape 1,344 -> 1,268, 8 x 128 prompts 618 -> 587)
                    float* dst = g.of + (size_t)row * g.nfeat + f;
#pragma unroll
                    for (int i = 0; i < CH; i++, dst += g.nfeat) add_f32(dst, v[i], i < m);
                } else if (EPI == EPI_GELU) {
                    u16* dst = g.oh + (size_t)row * g.pitch + f;
                    if (BM == 64 && g.rp) {
                        const size_t lo = (size_t)g.rp * g.pitch;
#pragma unroll
                        for (int i = 0; i < CH; i += 2, dst += 2 * g.pitch) {
                            const u32 h = pack_h2(v[i], v[i + 1]), r = pack_h2(v[i] - h_lo(h), v[i + 1] - h_hi(h));
                            st_u16(dst, (u16)h, i < m); st_u16(dst + g.pitch, (u16)(h >> 16), i + 1 < m);
                            st_u16(dst + lo, (u16)r, i < m); st_u16(dst + lo + g.pitch, (u16)(r >> 16), i + 1 < m);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < CH; i += 2, dst += 2 * g.pitch) {
                            const u32 h = pack_h2(v[i], v[i + 1]);
                            st_u16(dst, (u16)h, i < m); st_u16(dst + g.pitch, (u16)(h >> 16), i + 1 < m);
                        }
                    }
                } else {
                    float* dst = g.of + (size_t)row * g.nfeat + f;
#pragma unroll
                    for (int i = 0; i < CH; i++) st_f32(dst + (size_t)i * g.nfeat, v[i], i < m && !skip);
                    // The warp's best feature of every row (the lowest among equal ones): the lanes exchange halves of their rows until
                    // each holds one row. With redux and ballot row by row they took half the kernel's time (256 rows: 51.5 -> 33.4 us, 64: 18.0 -> 14.3).
                    int best[CH], at[CH];
#pragma unroll
                    for (int i = 0; i < CH; i++) {
                        best[i] = __float_as_int(v[i]);
                        best[i] = !own ? (int)0x80000000 : best[i] >= 0 ? best[i] : best[i] ^ 0x7fffffff;   // (below every logit, minus infinity included)
                        at[i] = lane;
                    }
                    int mine = 0;
#pragma unroll
                    for (int by = 16, w = CH / 2; by; by >>= 1, w >>= 1) {
                        const bool up = lane & by;
#pragma unroll
                        for (int i = 0; i < (w ? w : 1); i++) {
                            const int keep = w && up ? best[i + w] : best[i], at_keep = w && up ? at[i + w] : at[i];
                            const int other = __shfl_xor_sync(0xffffffffu, w && !up ? best[i + w] : best[i], by);
                            const int at_other = by == 16 ? lane ^ 16 : __shfl_xor_sync(0xffffffffu, w && !up ? at[i + w] : at[i], by);
                            const bool take = other > keep || (other == keep && at_other < at_keep);
                            best[i] = take ? other : keep;
                            at[i] = take ? at_other : at_keep;
                        }
                        if (up) mine += w;
                    }
                    if ((lane & (32 / CH - 1)) == 0) side[quarter * bn + c0 + mine] = f - lane + at[0] < g.nfeat && (AM == 128 || at[0] < 16) ? best_key(best[0], (u32)(f - lane + at[0])) : 0ull;
                }
            };
            int c0 = c_lo;
#pragma unroll 1
            for (; c0 + 8 < c_hi; c0 += 16) rows_of(Int<16>{}, c0);
            if (c0 + 4 < c_hi) rows_of(Int<8>{}, c0);
            else if (c0 < c_hi) rows_of(Int<4>{}, c0);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (PAIR) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(of_first(tme + b * 8)) : "memory");
                else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(tme + b * 8) : "memory");
            }
            if (EPI == EPI_LOGITS) {
                asm volatile("bar.sync 1, %0;" :: "n"(EW * 32) : "memory");
                if (!skip)
                    for (int i = et; i < live; i += EW * 32) {
                        u64 k = side[i];
#pragma unroll
                        for (int x = 1; x < 4; x++) if (side[x * bn + i] > k) k = side[x * bn + i];
                        if (k) atomicMax(g.best + row0 + i, k);
                    }
                if (two) asm volatile("bar.sync 1, %0;" :: "n"(EW * 32) : "memory");
            }
        }
        if (!waited) dep_wait();
    }
    __syncthreads();
    if (PAIR) cluster_sync();                                                      // (neither block leaves while the other may still reach into it)
    if (warp == 1) {
        if (*dead) settle();                                                       // (of a pair: both or none)
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(cols) : "memory");
    }
}

// ---- norm: (embedding,) LayerNorm, operand ---------------------------------------------------------------------------
#define PARTS_MAX 12                  // most parts of a cut fold
enum { NORM_EMBED = 0, NORM_MID = 1, NORM_FINAL = 2 };
struct NormArgs {
    int D, rp;
    float eps;
    float* z;                        // residual stream [row][D], updated in place
    const u16 *gain, *shift;
    u16* act;                        // [row][D] fp16 (and the remainder plane rp rows further)
    // EMBED: tokens and positions
    const int *x, *t, *seq;
    int t_stride, N, cpos, tmax, L;
    const u16 *wte, *wpe;
    long long* rowoff;
    int *pos, *skip;
    u32* bar;                        // [0] status, [2] abort flag
    const int* want;                 // FINAL: rows that want logits (0: all)
    const void* more;                // FINAL: a vector to add to the state (0: none)
    int fixed;                       // ... and both are State<true>
};

// One row per block, four elements per thread (the row stays in registers). Latency bound for few rows:
// mean and variance cost one exchange through shared memory: every warp
// takes the mean and the squared deviations of its own elements, the block combines them (Chan's formula).
template <int MODE>
__global__ void __launch_bounds__(1024) pass_norm(const __grid_constant__ NormArgs a) {
    __shared__ float2 red[32];
    const int tid = threadIdx.x, d = tid * 4, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const bool own = d < a.D;
    if (tid == 0) dep_launch();
    uint2 gw = make_uint2(0, 0), sw = make_uint2(0, 0);
    if (own) {
        gw = __ldg(reinterpret_cast<const uint2*>(a.gain + d)); sw = __ldg(reinterpret_cast<const uint2*>(a.shift + d));
    }
    const float rd = 1.0f / (float)a.D, rl = 1.0f / (float)(a.D - (nw - 1) * 128);   // one over the elements of the row, of the last warp
    if (MODE != NORM_EMBED) dep_wait();
    const int out = blockIdx.x;
    int row = out;
    if (MODE == NORM_FINAL && a.want) row = __ldg(a.want + out);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE == NORM_EMBED) {
        // tokens and positions outside their ranges would index outside the tables and the caches: the pass is refused
        // (a negative position: a sequence that has not started, its row is carried along and writes no cache)
        const int x = __ldcg(a.x + row), t = __ldcg(a.t + row * a.t_stride), sq = a.seq ? __ldcg(a.seq + row) : row;
        const bool aborted = __ldcg(a.bar + 2) != 0u;
        const bool bad = t >= a.tmax || t >= a.cpos || x < 0 || x >= a.N || aborted;
        if (tid == 0) {
            if (bad) { atomicExch(a.skip, 1); atomicCAS(a.bar, 0u, 0x900u); atomicExch(a.bar + 2, 1u); }
            a.rowoff[row] = (bad || t < 0) ? -1ll : ((long long)sq * a.L * a.tmax + t) * a.D;
            a.pos[row] = bad ? -1 : t;
        }
        if (own) {
            const uint2 e = __ldg(reinterpret_cast<const uint2*>(a.wte + (size_t)(bad ? 0 : x) * a.D + d)), p = __ldg(reinterpret_cast<const uint2*>(a.wpe + (size_t)(bad ? 0 : max(t, 0)) * a.D + d));
            v = make_float4(h_lo(e.x) + h_lo(p.x), h_hi(e.x) + h_hi(p.x), h_lo(e.y) + h_lo(p.y), h_hi(e.y) + h_hi(p.y));
        }
    } else if (own) {
        const size_t at = (size_t)row * a.D + d;
        if (MODE == NORM_FINAL && a.more) v = a.fixed ? State<true>::load(a.z, a.more, at) : State<false>::load(a.z, a.more, at);
        else v = State<false>::load(a.z, at);
    }
    if (own && MODE == NORM_EMBED) *reinterpret_cast<float4*>(a.z + (size_t)row * a.D + d) = v;
    float s = (v.x + v.y) + (v.z + v.w);
#pragma unroll
    for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    const float mw = s * (warp < nw - 1 ? 1.0f / 128.0f : rl);
    float y0 = v.x - mw, y1 = v.y - mw, y2 = v.z - mw, y3 = v.w - mw;
    float q = own ? (y0 * y0 + y1 * y1) + (y2 * y2 + y3 * y3) : 0.f;
#pragma unroll
    for (int m = 16; m; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    if (lane == 0) red[warp] = make_float2(s, q);
    __syncthreads();
    // the block's mean, then its squared deviations: every warp's own plus its elements times (its mean - the mean)^2
    const float2 mine = lane < nw ? red[lane] : make_float2(0.f, 0.f);
    s = mine.x;
#pragma unroll
    for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    const float mean = s * rd;
    const float dm = mine.x * (lane < nw - 1 ? 1.0f / 128.0f : rl) - mean;
    q = lane < nw ? mine.y + (lane < nw - 1 ? 128.0f : (float)(a.D - (nw - 1) * 128)) * dm * dm : 0.f;
#pragma unroll
    for (int m = 16; m; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    const float rs = rsqrtf(q * rd + a.eps);
    if (own) {
        const float o0 = (v.x - mean) * rs * h_lo(gw.x) + h_lo(sw.x), o1 = (v.y - mean) * rs * h_hi(gw.x) + h_hi(sw.x);
        const float o2 = (v.z - mean) * rs * h_lo(gw.y) + h_lo(sw.y), o3 = (v.w - mean) * rs * h_hi(gw.y) + h_hi(sw.y);
        const u32 p0 = pack_h2(o0, o1), p1 = pack_h2(o2, o3);
        *reinterpret_cast<uint2*>(a.act + (size_t)out * a.D + d) = make_uint2(p0, p1);
        if (a.rp) *reinterpret_cast<uint2*>(a.act + (size_t)(a.rp + out) * a.D + d) = make_uint2(pack_h2(o0 - h_lo(p0), o1 - h_hi(p0)), pack_h2(o2 - h_lo(p1), o3 - h_hi(p1)));
    }
}

// The same for many rows: a warp per row, NV float4 per lane (8 rows of 768 floats per block; one row per block took 23 us for
// 9,200 rows, 1.8 TB/s).
template <int NV>
__global__ void __launch_bounds__(256) pass_norm_rows(const __grid_constant__ NormArgs a, int rows) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (threadIdx.x == 0) dep_launch();
    dep_wait();
    if (row >= rows) return;
    float* z = a.z + (size_t)row * a.D;
    float4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) { const int d = i * 128 + lane * 4; v[i] = d < a.D ? __ldcg(reinterpret_cast<const float4*>(z + d)) : make_float4(0.f, 0.f, 0.f, 0.f); }
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; i++) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
#pragma unroll
    for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    const float mean = s / a.D;
#pragma unroll
    for (int i = 0; i < NV; i++)
        if (i * 128 + lane * 4 < a.D) { v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean; q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w); }
#pragma unroll
    for (int m = 16; m; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    const float rs = rsqrtf(q / a.D + a.eps);
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int d = i * 128 + lane * 4;
        if (d < a.D) {
            const uint2 gw = __ldg(reinterpret_cast<const uint2*>(a.gain + d)), sw = __ldg(reinterpret_cast<const uint2*>(a.shift + d));
            *reinterpret_cast<uint2*>(a.act + (size_t)row * a.D + d) = make_uint2(pack_h2(v[i].x * rs * h_lo(gw.x) + h_lo(sw.x), v[i].y * rs * h_hi(gw.x) + h_hi(sw.x)),
                                                                                 pack_h2(v[i].z * rs * h_lo(gw.y) + h_lo(sw.y), v[i].w * rs * h_hi(gw.y) + h_hi(sw.y)));
        }
    }
}

// ---- attention of one position per row (decode) -----------------------------------------------------------------------
struct AttArgs {
    const float* q;                  // [row][D] fp32
    const u16 *kc, *vc;              // the caches at this layer
    long long seq_stride;            // elements between two sequences
    const int* t;                    // positions as the step began (they change only after it)
    int t_stride, tmax, D, pow2, rp;
    float scale;
    u16* out;                        // [row][D] fp16 (and the remainder plane)
};
__device__ __forceinline__ int kv_off(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ void cp16(u32 dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void ldsm4(u32 (&r)[4], u32 p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(p) : "memory");
}
__device__ __forceinline__ void ldsm4t(u32 (&r)[4], u32 p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(p) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const u32 (&a)[4], u32 b0, u32 b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Block = one (row, head), or half its positions where two blocks form a cluster (C = 2); warps take runs of 16 positions in
// turn, on mma.sync: scores = K rows (16 positions x 16 dims per step) times the query, its fp16 head in column 0 and its fp16
// remainder in column 1 (their sum is the fp32-accurate product); output = V transposed times the weights, head and remainder
// again in two columns. The same in fp32 on the ordinary cores took 14 instructions per position and head, most of them
// conversions of K and V, and was bound by them: 64 sequences of 512 positions 13.7 us per layer even with the cache in
// L2. A warp's next NS runs are on their way into shared memory (the L1 cache is small beside the contractions'
// blocks). The rows before the current position are there since earlier steps: the first NS runs are requested before the block
// waits for the kernel that computes the query and the current position's row.
#define ATT_RUN 16
__device__ __forceinline__ void cp16z(u32 dst, const void* src, bool yes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(yes ? 16 : 0) : "memory");
}
// One warp's runs of a row's positions: from `p0`, every `step`, through its ring of NS stages of 4 KB. request_first() asks for
// what is there since earlier steps, run() waits for nothing but that and leaves the 64 sums, the maximum and the sum of the weights
// in `part`; run(false) does one round of the same on what there is (a dry pass, see pass_few.cuh).
template <int NS> struct AttRow {
    const AttArgs& a;
    int row, h, first, step, n;
    u32 ring;
    const u16 *kp, *vp;
    u32 put[4];
    __device__ __forceinline__ AttRow(const AttArgs& args, int row_, int h_, int p0, int step_, u32 ring_) : a(args), row(row_), h(h_), first(p0), step(step_), ring(ring_) {
        const int lane = threadIdx.x & 31, pl = lane >> 3, dl = lane & 7;
        n = min(__ldcg(a.t + row * a.t_stride) + 1, a.tmax);
        kp = a.kc + row * a.seq_stride + h * 64 + dl * 8;
        vp = a.vc + row * a.seq_stride + h * 64 + dl * 8;
        // per stage 16 rows of K, then of V, 128 bytes each; the 16-byte pieces of a row swizzled (kv_off)
#pragma unroll
        for (int j = 0; j < 4; j++) put[j] = ring + kv_off(j * 4 + pl, dl);
    }
    __device__ __forceinline__ void request(int st, int p, int end) const {
        const int pl = (threadIdx.x & 31) >> 3;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int x = p + j * 4 + pl;
            const size_t off = (size_t)(x < end ? x : 0) * a.D;
            cp16z(put[j] + st * 4096, kp + off, x < end);
            cp16z(put[j] + st * 4096 + 2048, vp + off, x < end);
        }
    }
    __device__ __forceinline__ void request_first() const {
#pragma unroll
        for (int i = 0; i < NS; i++) {
            if (first + i * step < n) request(i, first + i * step, n - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
    __device__ __forceinline__ void run(bool real, float* part) const {
        const int lane = threadIdx.x & 31, pl = lane >> 3, dl = lane & 7, g = lane >> 2, t4 = lane & 3;
        int p0 = first;
        u32 bq[4][2];
        {
            const float* qp = a.q + (size_t)row * a.D + h * 64;
            float2 x[4][2];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                x[k][0] = __ldcg(reinterpret_cast<const float2*>(qp + k * 16 + 2 * t4));
                x[k][1] = __ldcg(reinterpret_cast<const float2*>(qp + k * 16 + 2 * t4 + 8));
            }
            // the current position, if it is in one of the runs requested above
            u32 at = 0;
#pragma unroll
            for (int i = 0; i < NS; i++) {
                const int y = n - 1 - (p0 + i * step);
                if (y >= 0 && y < ATT_RUN && (y & 3) == pl) at = ring + i * 4096 + kv_off(y, dl);
            }
            if (at) {
                const uint4 kc = __ldcg(reinterpret_cast<const uint4*>(kp + (size_t)(n - 1) * a.D)), vc = __ldcg(reinterpret_cast<const uint4*>(vp + (size_t)(n - 1) * a.D));
                asm volatile("cp.async.wait_all;" ::: "memory");                       // (the zeros that were requested in its place)
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(at), "r"(kc.x), "r"(kc.y), "r"(kc.z), "r"(kc.w) : "memory");
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(at + 2048), "r"(vc.x), "r"(vc.y), "r"(vc.z), "r"(vc.w) : "memory");
            }
            const float sc = a.pow2 ? 1.0f / a.scale : 1.0f;
#pragma unroll
            for (int k = 0; k < 4; k++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float u = x[k][i].x * sc, v = x[k][i].y * sc;
                    const u32 hi = pack_h2(u, v);
                    bq[k][i] = g & 1 ? pack_h2(u - h_lo(hi), v - h_hi(hi)) : hi;   // (every pair of columns alike: all lanes get scores)
                }
        }
        float m = -3.0e38f, den = 0.f, o[4][4];              // o[mt]: dims mt*16 + g (regs 0 + 1) and mt*16 + g + 8 (regs 2 + 3), lanes with t4 == 0
#pragma unroll
        for (int i = 0; i < 4; i++) { o[i][0] = 0.f; o[i][1] = 0.f; o[i][2] = 0.f; o[i][3] = 0.f; }
        int st = 0;
        const u32 ka = ring + kv_off(lane & 15, 0), va = ring + 2048 + ((lane & 7) + ((lane >> 4) ? 8 : 0)) * 128;
        const int kx = lane >> 4, k7 = lane & 7, vx = (lane >> 3) & 1;
#pragma unroll 1
        while (p0 < n) {
            asm volatile("cp.async.wait_group %0;" :: "n"(NS - 1) : "memory");
            __syncwarp();
            const u32 so = st * 4096;
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                u32 r[4];
                ldsm4(r, (ka & ~127u) + so + (((k * 2 + kx) ^ k7) << 4));
                mma16816(s, r, bq[k][0], bq[k][1]);
            }
            float s0 = s[0] + s[1], s1 = s[2] + s[3];        // positions p0 + g and p0 + g + 8
            if (!a.pow2) { s0 /= a.scale; s1 /= a.scale; }
            if (p0 + g >= n) s0 = -3.0e38f;
            if (p0 + g + 8 >= n) s1 = -3.0e38f;
            // (shuffles over the eight groups: redux took longer, 16 sequences of the XL shape 1,359 -> 1,344 us per step)
            float mx = fmaxf(s0, s1);
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            if (mx > m) {                                    // (the same in the whole warp)
                const float corr = fast_exp(m - mx);
                m = mx;
                den *= corr;
#pragma unroll
                for (int i = 0; i < 4; i++) { o[i][0] *= corr; o[i][1] *= corr; o[i][2] *= corr; o[i][3] *= corr; }
            }
            const float pa = s0 > -1.0e38f ? fast_exp(s0 - m) : 0.f, pb = s1 > -1.0e38f ? fast_exp(s1 - m) : 0.f;
            den += pa + pb;
            // the weights as operand: lane (g, t4) holds positions 2 t4, 2 t4 + 1 (and + 8); that of position r < 8 is `pa` of lane 4 r
            const float w00 = __shfl_sync(0xffffffffu, pa, 8 * t4), w01 = __shfl_sync(0xffffffffu, pa, 8 * t4 + 4);
            const float w10 = __shfl_sync(0xffffffffu, pb, 8 * t4), w11 = __shfl_sync(0xffffffffu, pb, 8 * t4 + 4);
            u32 b0 = pack_h2(w00, w01), b1 = pack_h2(w10, w11);
            if (g == 1) { b0 = pack_h2(w00 - h_lo(b0), w01 - h_hi(b0)); b1 = pack_h2(w10 - h_lo(b1), w11 - h_hi(b1)); }
            if (g > 1) { b0 = 0; b1 = 0; }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                u32 r[4];
                ldsm4t(r, va + so + (((i * 2 + vx) ^ k7) << 4));
                mma16816(o[i], r, b0, b1);
            }
            __syncwarp();                                    // every lane has read the stage
            if (!real) break;
            if (p0 + NS * step < n) request(st, p0 + NS * step, n);
            asm volatile("cp.async.commit_group;" ::: "memory");
            p0 += step;
            if (++st == NS) st = 0;
        }
#pragma unroll
        for (int x = 16; x > 2; x >>= 1) den += __shfl_xor_sync(0xffffffffu, den, x);
        if (t4 == 0)
#pragma unroll
            for (int i = 0; i < 4; i++) { part[i * 16 + g] = o[i][0] + o[i][1]; part[i * 16 + g + 8] = o[i][2] + o[i][3]; }
        if (lane == 0) { part[64] = m; part[65] = den; }
    }
};
template <int NS, int W>
__global__ void __launch_bounds__(W * 32) pass_attend(const __grid_constant__ AttArgs a) {
    __shared__ float part[W + 1][66];
    extern __shared__ __align__(128) unsigned char ring_raw[];
    const int h = blockIdx.x, row = blockIdx.y, C = gridDim.z, cr = blockIdx.z, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) dep_launch();
    if (C == 2) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // (waited for before the other block's memory is written)
    AttRow<NS> r(a, row, h, (cr * W + warp) * ATT_RUN, C * W * ATT_RUN, smem_u32(ring_raw) + warp * (NS * 4096));
    r.request_first();
    dep_wait();
    r.run(true, part[warp]);
    __syncthreads();
    float M = -3.0e38f, dd = 0.f, num = 0.f;
    if (threadIdx.x < 64) {
#pragma unroll
        for (int i = 0; i < W; i++) M = fmaxf(M, part[i][64]);
#pragma unroll
        for (int i = 0; i < W; i++) { const float c = fast_exp(part[i][64] - M); dd += part[i][65] * c; num += part[i][threadIdx.x] * c; }
    }
    if (C == 2) {
        // the second block's result goes into the first one's shared memory
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (cr == 1 && threadIdx.x < 64) {
            const u32 to = of_first(smem_u32(&part[W][0]));
            asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(to + threadIdx.x * 4), "f"(num) : "memory");
            if (threadIdx.x == 0) asm volatile("st.shared::cluster.f32 [%0], %1;\n\tst.shared::cluster.f32 [%0+4], %2;" :: "r"(to + 64 * 4), "f"(M), "f"(dd) : "memory");
        }
        cluster_sync();
        if (cr == 1) return;
        if (threadIdx.x < 64) {
            const float m1 = part[W][64], top = fmaxf(M, m1), c0 = fast_exp(M - top), c1 = fast_exp(m1 - top);
            dd = dd * c0 + part[W][65] * c1;
            num = num * c0 + part[W][threadIdx.x] * c1;
        }
    }
    if (threadIdx.x < 64) {
        const float r = dd > 0.f ? __fdividef(num, dd) : 0.f;                      // a sequence that has not started attends to nothing
        const u16 hi = f2h(r);
        a.out[(size_t)row * a.D + h * 64 + threadIdx.x] = hi;
        if (a.rp) a.out[(size_t)(a.rp + row) * a.D + h * 64 + threadIdx.x] = f2h(r - h2f(hi));
    }
}

// ---- attention of many positions (prompts) ----------------------------------------------------------------------------
struct AttManyArgs {
    const int4* tiles;               // (first row, rows, sequence, first position) of every run of at most 128 rows of one sequence
    int layer, L, D;
    float scale;
    u16* out;                        // [row][D] fp16
    u32* status;
    u64 limit;                       // of a wait, ns
};
__device__ __forceinline__ void tm_ld32(u32 (&r)[32], u32 addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
                   "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]) : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                   "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]) : : "memory");
    asm volatile("" : "+r"(r[30]), "+r"(r[31]));
}
__device__ __forceinline__ void tm_st32(u32 addr, const u32 (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
                 :: "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                    "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
                    "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(addr) : "memory");
}
#define AM_STAGES 2
#define AM_SMEM (32768 + AM_STAGES * 32768 + 128 + 2048 + 1024)
#define AM_THREADS 320
// Block = up to 128 consecutive positions of one sequence x one head; the cache in tiles of 128 positions; causal. On tcgen05:
// scores = queries (fp16 head and remainder from the QKV contraction, two products: fp32 accuracy over the fp16 cache) x K rows, 128 x 128 in tensor
// memory; two threads own a row, 32 columns in turn, and exchange its maximum; the weights go back into the columns of the
// scores as fp16 head and remainder (operand A of the second product, in tensor memory) x V rows (N-major as they lie in the
// cache). The output is rescaled only when a row's maximum has grown by more than 5.5 (the weights stay below 2^8, and the
// same maximum normalises them at the end). Two blocks per SM: one's exponentials run under the other's products.
// At 9,200 rows of 32 prompts of 64 to 512 a layer took 58 us with mma.sync (64 rows per block, the same two-part operands;
// bound by the products), 39 with one thread per row and queries read as fp32, 35 now, of which the products are 9: a block
// is a chain of load, products, exponentials, products, and two fit an SM. 77 positions: 5.7 -> 4.6 us.
template <bool POW2>                                    // the divisor of the scores is a power of two: applied to the queries
__global__ void __launch_bounds__(AM_THREADS, 2) pass_attend_many(const __grid_constant__ CUtensorMap qm, const __grid_constant__ CUtensorMap km, const __grid_constant__ CUtensorMap vm, const __grid_constant__ AttManyArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const u32 sq = smem_u32(smem), skv = sq + 32768, bars = skv + AM_STAGES * 32768;
    const u32 qf = bars, sf = bars + 8, pf = bars + 16, of = bars + 24, kvf = bars + 32, kve = kvf + AM_STAGES * 8;
    unsigned char* tail = smem + 32768 + AM_STAGES * 32768 + 32 + AM_STAGES * 16;
    volatile u32* tmem_p = reinterpret_cast<volatile u32*>(tail);
    volatile int* dead = reinterpret_cast<volatile int*>(tail + 4);
    float* pair = reinterpret_cast<float*>(tail + 16);                             // [tile & 1][half][row]: maxima, at the end sums
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const Wait w{smem_u32(tail + 4), 0u, a.status, a.limit};
    if (threadIdx.x == 0) {
        *dead = 0;
        mbar_init(qf, 1); mbar_init(sf, 1); mbar_init(pf, 8); mbar_init(of, 1);
        for (int i = 0; i < AM_STAGES; i++) { mbar_init(kvf + i * 8, 1); mbar_init(kve + i * 8, 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&qm) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&km) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(&vm) : "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tail)), "n"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (threadIdx.x == 0) dep_launch();
    const u32 tmem = *tmem_p, tO = tmem + 128;                                     // scores / weights: columns 0..127, output: 128..191
    const int4 tl = __ldg(a.tiles + blockIdx.y);                                   // (runs in the order of their work, all heads of one before the next)
    const int h = blockIdx.x, row0 = tl.x, nrows = tl.y, pos0 = tl.w, total = pos0 + nrows, nt = (total + 127) / 128;
    if (warp == 8) {
        if (elect_one()) {
            dep_wait();
            mbar_expect(qf, 32768);
            tma3(sq, &qm, h * 64, row0, 0, qf);
            tma3(sq + 16384, &qm, h * 64, row0, 1, qf);
            for (int j = 0; j < nt; j++) {
                const int s = j % AM_STAGES;
                if (j >= AM_STAGES && !mbar_wait(kve + s * 8, (j / AM_STAGES - 1) & 1, w, 0xC00u)) break;
                const u32 dst = skv + s * 32768;
                mbar_expect(kvf + s * 8, 32768);
                tma3(dst, &km, h * 64, j * 128, tl.z * a.L + a.layer, kvf + s * 8);
                tma3(dst + 16384, &vm, h * 64, j * 128, tl.z * a.L + a.layer, kvf + s * 8);
            }
        }
    } else if (warp == 9) {
        constexpr u32 i_s = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24), i_o = (1u << 4) | (1u << 16) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
        bool ok = !__any_sync(0xffffffffu, !mbar_wait(qf, 0, w, 0xC10u));
        for (int j = 0; j < nt && ok; j++) {
            const int s = j % AM_STAGES;
            ok = !__any_sync(0xffffffffu, !mbar_wait(kvf + s * 8, (j / AM_STAGES) & 1, w, 0xC20u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const u64 q = desc_k(sq), k = desc_k(skv + s * 32768);
#pragma unroll
                for (int i = 0; i < 8; i++)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                 :: "r"(tmem), "l"(q + (i >> 2) * 1024 + 2 * (i & 3)), "l"(k + 2 * (i & 3)), "r"(i_s), "r"(i ? 1u : 0u) : "memory");
                tc_commit<false>(sf);
            }
            __syncwarp();
            ok = !__any_sync(0xffffffffu, !mbar_wait(pf, j & 1, w, 0xC30u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const u64 v = desc_m(skv + s * 32768 + 16384, 8192);
                const int nk = min(8, (total - j * 128 + 15) / 16);                // steps of 16 positions that some row sees
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k < nk) {
#pragma unroll
                        for (int x = 0; x < 2; x++)
                            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                                         :: "r"(tO), "r"(tmem + (k >> 1) * 32 + (k & 1) * 8 + x * 16), "l"(v + 128 * k), "r"(i_o), "r"((j | k | x) ? 1u : 0u) : "memory");
                    }
                tc_commit<false>(kve + s * 8);
                if (j == nt - 1) tc_commit<false>(of);
            }
            __syncwarp();
        }
    } else {
        const int quad = warp & 3, half = warp >> 2;                               // two threads per row: 32 columns of the scores in turn
        const int row = quad * 32 + lane, p = pos0 + row;                          // this thread's row of the tile, its position
        const u32 mine = (u32)(quad * 32) << 16;
        constexpr float LOG2E = 1.4426950408889634f;
        float m = -3.0e38f, den = 0.f;
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < nt; j++) {
            if (ok) ok = !__any_sync(0xffffffffu, !mbar_wait(sf, j & 1, w, 0xC40u));
            if (!ok) {                                                             // (the other warp of these rows may not have given up)
                asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
                continue;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int lim = p - j * 128;                                           // last column of the tile that this row sees
            const int chunks = min(4, (total - j * 128 + 31) / 32);                // chunks of 32 columns that the second product reads,
            const int seen = max(0, min(chunks, (lim - lane + 31) / 32 + (lim - lane + 31 >= 0 ? 1 : 0)));   // and that some row of this warp sees
            u32 r[32];
            // (chunks that all rows of the warp see whole carry no mask: 7 instead of 11 instructions per score)
            const int whole = min(seen, (lim - lane + 1) >> 5);
            float top[4] = {-3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f};
            auto maxima = [&](auto MASK, int c) {
                tm_ld32(r, tmem + mine + c * 32);
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    float s = __uint_as_float(r[i]);
                    if (!POW2) s /= a.scale;
                    if (decltype(MASK)::n) s = c * 32 + i <= lim ? s : -3.0e38f;
                    top[i & 3] = fmaxf(top[i & 3], s);
                }
            };
            int c = half;
#pragma unroll 1
            for (; c < whole; c += 2) maxima(Int<0>{}, c);
#pragma unroll 1
            for (; c < seen; c += 2) maxima(Int<1>{}, c);
            float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            pair[(j & 1) * 256 + half * 128 + row] = mx;
            asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
            mx = fmaxf(mx, pair[(j & 1) * 256 + (half ^ 1) * 128 + row]);
            const bool grow = mx > m + 5.5f;
            if (__any_sync(0xffffffffu, grow)) {
                const float corr = grow ? fast_exp(m - mx) : 1.0f;
                if (grow) m = mx;
                den *= corr;
                if (j > 0) {                                                       // (the products into the output have completed: the scores' came after them)
                    tm_ld32(r, tO + mine + half * 32);
#pragma unroll
                    for (int i = 0; i < 32; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
                    tm_st32(tO + mine + half * 32, r);
                }
            }
            const float m2 = m * LOG2E;
            auto weights = [&](auto MASK, int c) {
                u32 o[32];
                float sum[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
                tm_ld32(r, tmem + mine + c * 32);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float e[2];
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        float s = __uint_as_float(r[i + x]);
                        if (!POW2) s /= a.scale;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e[x]) : "f"(fmaf(s, LOG2E, -m2)));
                        if (decltype(MASK)::n) e[x] = c * 32 + i + x <= lim ? e[x] : 0.f;
                        sum[(i / 2) & 1][x] += e[x];
                    }
                    o[i / 2] = pack_h2(e[0], e[1]);
                    o[16 + i / 2] = pack_h2(e[0] - h_lo(o[i / 2]), e[1] - h_hi(o[i / 2]));
                }
                den += (sum[0][0] + sum[0][1]) + (sum[1][0] + sum[1][1]);
                tm_st32(tmem + mine + c * 32, o);
            };
#pragma unroll 1
            for (c = half; c < whole; c += 2) weights(Int<0>{}, c);
#pragma unroll 1
            for (; c < seen; c += 2) weights(Int<1>{}, c);
#pragma unroll 1
            for (; c < chunks; c += 2) {
#pragma unroll
                for (int i = 0; i < 32; i++) r[i] = 0u;
                tm_st32(tmem + mine + c * 32, r);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(pf) : "memory");
        }
        if (ok) ok = !__any_sync(0xffffffffu, !mbar_wait(of, 0, w, 0xC50u));
        if (!ok) asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
        else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // (every row has waited for the last products, which came after all reads of the maxima)
            pair[half * 128 + row] = den;
            asm volatile("bar.sync %0, 64;" :: "r"(1 + quad) : "memory");
            den += pair[(half ^ 1) * 128 + row];
            const float inv = den > 0.f ? __fdividef(1.0f, den) : 0.f;
            uint4* out = reinterpret_cast<uint4*>(a.out + (size_t)(row0 + row) * a.D + h * 64 + half * 32);
            u32 r[32];
            tm_ld32(r, tO + mine + half * 32);
            if (row < nrows)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float* v = reinterpret_cast<const float*>(r) + i * 8;
                    out[i] = make_uint4(pack_h2(v[0] * inv, v[1] * inv), pack_h2(v[2] * inv, v[3] * inv), pack_h2(v[4] * inv, v[5] * inv), pack_h2(v[6] * inv, v[7] * inv));
                }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
    }
    __syncthreads();
    if (warp == 9) {
        if (*dead) settle();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(256) : "memory");
    }
}

// ---- the end of a pass: the chosen tokens, feedback ---------------------------------------------------------------------
struct FinishArgs {
    int rows;
    u64* best;
    int* skip;
    const u32* bar;                  // [2] abort flag
    float* next;                     // decode: the chosen tokens as float (0: none)
    const int* pos;
    int *x, *t;                      // fed back (0: no feedback)
    int t_stride, tstep, N;
    const int *prompt, *plen;
    int plen_cap;
    const int2* dst;                 // prompts: sequence of the row, length of its prompt
};
__global__ void __launch_bounds__(256) pass_finish(const __grid_constant__ FinishArgs a) {
    dep_wait();
    const bool skip = __ldcg(a.skip) != 0 || __ldcg(a.bar + 2) != 0u;
    for (int b = threadIdx.x; b < a.rows; b += blockDim.x) {
        const u64 k = __ldcg(a.best + b);
        a.best[b] = 0ull;
        if (skip) continue;
        const u32 n = 0xFFFFFFFFu - (u32)(k & 0xFFFFFFFFull);
        if (a.next) a.next[b] = (float)n;
        if (a.dst) {
            const int2 e = __ldg(a.dst + b);
            a.x[e.x] = (n >= (u32)a.N) ? 0 : (int)n;
            a.t[e.x * a.t_stride] = e.y;
            continue;
        }
        if (a.x) {
            int nx = (int)n;
            const int tn = a.pos[b] + a.tstep;
            if (a.plen && tn >= 0 && tn < a.plen[b]) nx = a.prompt[(size_t)b * a.plen_cap + tn];
            a.x[b] = (nx < 0 || nx >= a.N) ? 0 : nx;
            if (a.t_stride || b == 0) a.t[b * a.t_stride] = tn;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) *a.skip = 0;
}

}  // namespace vesta_pass
