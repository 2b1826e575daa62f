// Kernels of a decode step of few sequences (two to four): three per layer,
//
//     norm + QKV | attention + projection | norm + FC + GELU + MLP projection
//
// then the last norm, the logits and the end of pass_kernels.cuh, launched with programmatic stream serialization like those.
//
// What bounds such a step is neither memory nor the tensor cores but the exchanges between the SMs and the chains of latencies
// between them: GPT-2 small has 14 MB of weights per layer, 2.2 us of memory traffic, and took 15 to 17 us per layer in one persistent
// kernel with grid barriers. So a kernel boundary (1.2 us) stands only where every SM needs sums of all the others: before the two
// norms and before the attention, and everything else stays within a block or a cluster of eight blocks:
//   * every block normalises all rows by itself, with two or four warps to a row (the state of four sequences is 12 KB);
//   * the eight blocks of a head exchange their attention results through distributed shared memory and each applies an eighth of
//     the head's rows of the projection to all sequences;
//   * a block keeps the GELU output of its own features and multiplies it with their rows of the MLP projection.
// Measured on B200 (small shape, 200 positions, steps of sixteen): two sequences 184 -> 168 us per step, three 186 -> 158, four 191 -> 163; per layer 12.9,
// 12.3 and 12.5 us, of which 3 to 4 are boundaries and the rest the kernels' own chains.
// The weights a block needs are on their way into its shared memory before it waits for its predecessor. They are a copy in the order
// in which the lanes of mma.sync m16n8k16 hold them, so that every thread copies (cp.async) and reads back just its own 16 bytes of
// each unit: no barrier, nothing to wait for but its own copies. The activations enter as fp16 head and remainder, whose products
// add up to the fp32-accurate one: the eight columns of operand B are sequence 0 head, remainder, sequence 1, ..., the rows of A 16 features.
// (One product takes 13 to 16 cycles of a quarter of an SM, a sixth of what tcgen05 could do; but that has 64 or 128 rows, and its
// operands would make two more trips through shared memory.)
#pragma once
#include "pass_kernels.cuh"

namespace vesta_pass {

// The dry pass: what a kernel does after its wait it does once before, on whatever is in its shared memory and without a store to
// global memory. Its instructions and parameters are then in the SM's caches when its input arrives: a kernel runs each of its
// instructions once or twice, and fetched one after the other from L2 they took longer than anything they do.
// (The compiler is not to know how often the loop runs, two copies of the code would warm nothing, and is not to move what both passes
// compute in front of it, which costs registers.)
__device__ __forceinline__ int few_passes(int n) { asm volatile("" : "+r"(n)); return n; }
#define FEW_ROWS 4
#define FEW_RED (FEW_ROWS * 16)          // a warp's sums of a tile
#define FEW_WARPS 8
#define FEW_THREADS (FEW_WARPS * 32)
#define FEW_CLUSTER 8                 // blocks of a head
#define FEW_TILES 2                   // most tiles of 16 features of a block
#define FEW_STAGES 2                  // stages of a warp's ring in the attention

// Packed weights of a layer, in units of 512 bytes, 16 per lane (g = lane / 4, t = lane % 4):
//   qkv, fc: [16 features][32 fold indices][2 units, one half of the fold indices each]
//   proj, p2: [16 outputs][16 fold indices]
// every unit as operand A: fold indices 2t, 2t+1 of features g, g+8, then 2t+8, 2t+9 of both
// proj: [head][16 outputs][4 units of the head's 64 fold indices]; p2: [16 fold indices][16 outputs]
struct FewPack {
    size_t qkv, proj, fc, p2, layer;          // offsets in a layer, bytes of a layer
    __host__ __device__ FewPack(int D, int F) {
        qkv = 0; proj = qkv + (size_t)3 * D * D * 2; fc = proj + (size_t)D * D * 2; p2 = fc + (size_t)D * F * 2; layer = p2 + (size_t)D * F * 2;
    }
};
struct FewPackArgs { int D, F, L; const u16 *qkvw, *ow, *fcw, *pw; unsigned char* out; };
// A warp takes 1 KB of qkv / fc or a unit of proj / p2 at a time: 16 bytes per lane and load, through shared memory into the lanes' order.
__global__ void __launch_bounds__(256) few_pack(const __grid_constant__ FewPackArgs a) {
    __shared__ __align__(16) u16 buf[8][32 * 24];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, D = a.D, F = a.F, KP = D / 32, MT = D / 16;
    u16* s = buf[warp];
    const FewPack off(D, F);
    const long long n1 = (long long)(3 * D / 16) * KP, n2 = (long long)(F / 16) * KP, n3 = (long long)MT * MT, n4 = (long long)(F / 16) * MT, per = n1 + n2 + n3 + n4;
    for (long long u = (long long)blockIdx.x * 8 + warp; u < per * a.L; u += (long long)gridDim.x * 8) {
        const long long l = u / per;
        long long i = u - l * per;
        unsigned char* out = a.out + (size_t)l * off.layer;
        u32 w[4];
        auto two = [&](int k, int o) { return (u32)s[k * 24 + o] | ((u32)s[(k + 1) * 24 + o] << 16); };
        __syncwarp();
        if (i < n1 + n2) {
            const bool fc = i >= n1;
            if (fc) i -= n1;
            const int ld = fc ? F : 3 * D, kp = (int)(i % KP), tile = (int)(i / KP);
            const u16* src = (fc ? a.fcw + (size_t)l * D * F : a.qkvw + (size_t)l * D * 3 * D) + (size_t)(kp * 32 + lane) * ld + tile * 16;
            *reinterpret_cast<uint4*>(s + lane * 24) = __ldg(reinterpret_cast<const uint4*>(src));
            *reinterpret_cast<uint4*>(s + lane * 24 + 8) = __ldg(reinterpret_cast<const uint4*>(src) + 1);
            __syncwarp();
            for (int j = 0; j < 2; j++) {
                for (int q = 0; q < 4; q++) w[q] = two(j * 16 + (q >> 1) * 8 + 2 * t, (q & 1) * 8 + g);
                *reinterpret_cast<uint4*>(out + (fc ? off.fc : off.qkv) + (((size_t)tile * KP + kp) * 2 + j) * 512 + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        } else {
            i -= n1 + n2;
            const bool p2 = i >= n3;
            if (p2) i -= n3;
            const int mt = (int)(i % MT), kt = (int)(i / MT);
            const u16* src = (p2 ? a.pw + (size_t)l * F * D : a.ow + (size_t)l * D * D) + (size_t)(kt * 16 + (lane >> 1)) * D + mt * 16 + (lane & 1) * 8;
            *reinterpret_cast<uint4*>(s + (lane >> 1) * 24 + (lane & 1) * 8) = __ldg(reinterpret_cast<const uint4*>(src));
            __syncwarp();
            for (int q = 0; q < 4; q++) w[q] = two((q >> 1) * 8 + 2 * t, (q & 1) * 8 + g);
            const size_t at = p2 ? off.p2 + ((size_t)kt * MT + mt) * 512 : off.proj + (((size_t)(kt >> 2) * MT + mt) * 4 + (kt & 3)) * 512;
            *reinterpret_cast<uint4*>(out + at + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// Operand rows in shared memory, `ld` bytes apart: heads and remainders in turn. Where a lane points ldmatrix for the first 32 fold
// indices; rows that do not exist repeat the last
__device__ __forceinline__ u32 few_row(u32 op, int ld, int R, int lane) { return op + min(lane & 7, 2 * R - 1) * ld + (lane >> 3) * 16; }
// a 16-byte piece of this thread's own weights
__device__ __forceinline__ uint4 lds16(u32 p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void few_mma(float (&c)[4], const uint4& a, u32 b0, u32 b1) {
    const u32 r[4] = {a.x, a.y, a.z, a.w};
    mma16816(c, r, b0, b1);
}
// the sums of a tile of outputs (proj, p2; c[0] and c[1]: parts of the same sums) into the state
template <bool FIXED> __device__ __forceinline__ void few_add(void* z, int D, int R, int tile, const float (&c)[2][4], int lane) {
    const int g = lane >> 2, t = lane & 3;
    if (t < R) {
        const size_t at = (size_t)t * D + tile * 16 + g;
        State<FIXED>::add1(z, at, (c[0][0] + c[0][1]) + (c[1][0] + c[1][1]));
        State<FIXED>::add1(z, at + 8, (c[0][2] + c[0][3]) + (c[1][2] + c[1][3]));
    }
}

// The state between two layers is a vector that the attention's projections have been added to, and one of the MLP's sums alone: sums of
// 96 parts that come in any order round at their own size, not at the state's.
struct FewNorm {
    int D, rows;
    float eps;
    const void *z, *more;             // [row][D]; QKV: their sum
    const u16 *gain, *shift;
    void* into;                       // the vector that the next sums go into: QKV: it starts as the state plus `bias`, MLP: as `bias`
    const u16* bias;
    void* clear;                      // QKV: the vector after that, zeroed
    static __host__ __device__ int bytes(int D) { return 3 * D * 2; }
};
// gain, shift and bias into shared memory, before the wait (which empties the L1 cache)
__device__ __forceinline__ void few_params(const FewNorm& n, u16* par) {
    for (int d = threadIdx.x * 4; d < n.D; d += FEW_THREADS * 4) {
        *reinterpret_cast<uint2*>(par + d) = __ldg(reinterpret_cast<const uint2*>(n.gain + d));
        *reinterpret_cast<uint2*>(par + n.D + d) = __ldg(reinterpret_cast<const uint2*>(n.shift + d));
        if (blockIdx.x < n.rows) *reinterpret_cast<uint2*>(par + 2 * n.D + d) = __ldg(reinterpret_cast<const uint2*>(n.bias + d));
    }
}
// Norm of all rows into the operand. WPR warps share a row (four of two rows, two of three or four), a lane holds NV float4. Block `row` (counted around where there are fewer) also starts the
// vector of the next sums: QKV stores it (nothing adds yet), the MLP kernel adds to it (other blocks may have begun to).
// `value(row, d)` loads four elements of the state.
template <int KW, int WPR> struct FewLanes { static constexpr int NV = (2 * KW + WPR - 1) / WPR; };      // KW: D <= 256 KW
template <int KW, int WPR, bool FIXED, bool STORE, class Load>
__device__ __forceinline__ void few_norm(const FewNorm& n, bool real, int warp, int lane, const u16* par, unsigned char* op, int ld, float2* red, Load value) {
    constexpr int NV = FewLanes<KW, WPR>::NV, by = WPR * 128;
    const int row = warp / WPR, seg = warp % WPR, d0 = (seg * 32 + lane) * 4;
    const bool live = row < n.rows;
    float4 v[NV];
    auto elements = [&](int x) {                                                   // of the row's warp x
        int c = 0;
#pragma unroll
        for (int i = 0; i < NV; i++) c += max(0, min(128, n.D - (x * 128 + i * by)));
        return c;
    };
    const float rd = 1.0f / (float)n.D, own = (float)elements(seg), rown = own > 0.f ? 1.0f / own : 0.f;
    const float cx = (float)elements(lane % WPR), rcx = cx > 0.f ? 1.0f / cx : 0.f;
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int d = d0 + i * by;
        v[i] = live && d < n.D ? value(row, d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < NV; i++) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
#pragma unroll
    for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    float mean = s * rown;
#pragma unroll
    for (int i = 0; i < NV; i++)
        if (d0 + i * by < n.D) {
            const float a = v[i].x - mean, b = v[i].y - mean, c = v[i].z - mean, e = v[i].w - mean;
            q += (a * a + b * b) + (c * c + e * e);
        }
#pragma unroll
    for (int m = 16; m; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    // the row's mean, then its squared deviations: every warp's own plus its elements times (its mean - the mean)^2
    if (lane == 0) red[warp] = make_float2(s, q);
    __syncthreads();
    const float2 p = red[row * WPR + lane % WPR];
    s = p.x;
#pragma unroll
    for (int m = WPR / 2; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    mean = s * rd;
    const float dm = p.x * rcx - mean;
    q = cx > 0.f ? p.y + cx * dm * dm : 0.f;
#pragma unroll
    for (int m = WPR / 2; m; m >>= 1) q += __shfl_xor_sync(0xffffffffu, q, m);
    const float rs = rsqrtf(q * rd + n.eps);
    if (live) {
        unsigned char *hi = op + 2 * row * ld, *lo = hi + ld;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int d = d0 + i * by;
            if (d < n.D) {
                const uint2 gw = *reinterpret_cast<const uint2*>(par + d), sw = *reinterpret_cast<const uint2*>(par + n.D + d);
                const float o0 = (v[i].x - mean) * rs * h_lo(gw.x) + h_lo(sw.x), o1 = (v[i].y - mean) * rs * h_hi(gw.x) + h_hi(sw.x);
                const float o2 = (v[i].z - mean) * rs * h_lo(gw.y) + h_lo(sw.y), o3 = (v[i].w - mean) * rs * h_hi(gw.y) + h_hi(sw.y);
                const u32 p0 = pack_h2(o0, o1), p1 = pack_h2(o2, o3);
                *reinterpret_cast<uint2*>(hi + d * 2) = make_uint2(p0, p1);
                *reinterpret_cast<uint2*>(lo + d * 2) = make_uint2(pack_h2(o0 - h_lo(p0), o1 - h_hi(p0)), pack_h2(o2 - h_lo(p1), o3 - h_hi(p1)));
            }
        }
        if (blockIdx.x == row % gridDim.x && real)
#pragma unroll
            for (int i = 0; i < NV; i++) {
                const int d = d0 + i * by;
                if (d < n.D) {
                    const uint2 b = *reinterpret_cast<const uint2*>(par + 2 * n.D + d);
                    const float4 sum = STORE ? make_float4(v[i].x + h_lo(b.x), v[i].y + h_hi(b.x), v[i].z + h_lo(b.y), v[i].w + h_hi(b.y)) : make_float4(h_lo(b.x), h_hi(b.x), h_lo(b.y), h_hi(b.y));
                    const size_t at = (size_t)row * n.D + d;
                    if (STORE) {
                        State<FIXED>::store(n.into, at, sum);
                        State<FIXED>::store(n.clear, at, make_float4(0.f, 0.f, 0.f, 0.f));
                    } else State<FIXED>::add(n.into, at, sum);
                }
            }
    }
}

// A warp takes every eighth pair of units of the fold of each tile; they lie one after the other in its own part of shared memory, KU
// pairs to a tile (zeros in the place of one that does not exist). Requests `n` tiles (KP pairs each from `w`).
__device__ __forceinline__ int few_units(int KP) { return (KP + FEW_WARPS - 1) / FEW_WARPS; }
__device__ __forceinline__ void few_request(u32 slots, const unsigned char* w, int n, int KP, int warp, int lane) {
    const int KU = few_units(KP);
    w += lane * 16;
    slots += lane * 16;
#pragma unroll 1
    for (int j = 0; j < n; j++, w += KP * 1024, slots += KU * 1024)
#pragma unroll 1
        for (int i = 0; i < KU; i++) {
            const int k = warp + i * FEW_WARPS;
            const unsigned char* src = w + (k < KP ? k : 0) * 1024;
            cp16z(slots + i * 1024, src, k < KP);
            cp16z(slots + i * 1024 + 512, src + 512, k < KP);
        }
}
// ... and multiplies them with the operand: red[tile][warp][row][16 features]
template <int KW>
__device__ __forceinline__ void few_fold(u32 slots, u32 a_at, int n, int KP, float* red, int warp, int lane) {
    const int KU = few_units(KP), g = lane >> 2, t = lane & 3;
    u32 a[KW][4];
#pragma unroll
    for (int i = 0; i < KW; i++) {
        const bool yes = warp + i * FEW_WARPS < KP;
        const u32 at = a_at + (yes ? warp + i * FEW_WARPS : 0) * 64;
        ldsm4(a[i], at);
        if (!yes)
#pragma unroll
            for (int x = 0; x < 4; x++) a[i][x] = 0u;
    }
    slots += lane * 16;
    red += warp * FEW_RED;
#pragma unroll 1
    for (int j = 0; j < n; j++) {
        float c[2][2][4] = {};
        uint4 w[KW][2];
#pragma unroll
        for (int i = 0; i < KW; i++) { w[i][0] = lds16(slots + (j * KU + min(i, KU - 1)) * 1024); w[i][1] = lds16(slots + (j * KU + min(i, KU - 1)) * 1024 + 512); }
#pragma unroll
        for (int i = 0; i < KW; i++) { few_mma(c[i & 1][0], w[i][0], a[i][0], a[i][1]); few_mma(c[i & 1][1], w[i][1], a[i][2], a[i][3]); }
        float* to = red + j * (FEW_WARPS * FEW_RED);
        // feature g (and g + 8) of row t: head and remainder are neighbours, four accumulators hold parts of the fold
        to[t * 16 + g] = ((c[0][0][0] + c[0][0][1]) + (c[0][1][0] + c[0][1][1])) + ((c[1][0][0] + c[1][0][1]) + (c[1][1][0] + c[1][1][1]));
        to[t * 16 + g + 8] = ((c[0][0][2] + c[0][0][3]) + (c[0][1][2] + c[0][1][3])) + ((c[1][0][2] + c[1][0][3]) + (c[1][1][2] + c[1][1][3]));
    }
}
// the sum of the warps' parts of output `o` of a block: tile o / 64, row o / 16 % 4, feature o % 16
__device__ __forceinline__ float few_sum(const float* red, int o) {
    const float* p = red + (o / FEW_RED) * (FEW_WARPS * FEW_RED) + o % FEW_RED;
    float s[FEW_WARPS];
#pragma unroll
    for (int i = 0; i < FEW_WARPS; i++) s[i] = p[i * FEW_RED];
    return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// ---- norm + QKV -------------------------------------------------------------------------------------------------------
// A tile of 16 features per block (two beyond 148 tiles): 144 blocks at width 768. Bound by its chain: state from L2, statistics, operand,
// products, exchange between the warps. 4.6 us at two sequences (whose state is twice as wide), 4.1 at four, a boundary included.
struct FewQkv {
    FewNorm n;
    const unsigned char* w;           // packed, of the layer
    const u16* bias;
    int tiles, per;                   // tiles of 16 features, tiles per block
    float* q;                         // [row][D]
    u16 *kc, *vc;                     // the caches at this layer
    long long seq_stride;
    const int *x, *t;
    int t_stride, tmax, cpos, N, first;
    const u16 *wte, *wpe;             // first layer: the rows are embeddings
    int *pos, *skip;
    u32* bar;
    static __host__ __device__ int bytes(int D, int rows, int per) { return per * ((D / 32 + 7) / 8) * 8192 + 2 * rows * (2 * D + 16) + per * FEW_WARPS * FEW_RED * 4 + FewNorm::bytes(D); }
};
template <int KW, int WPR, bool FIXED>
__global__ void __launch_bounds__(FEW_THREADS, 2) few_qkv(const __grid_constant__ FewQkv a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float2 stat[FEW_WARPS];
    __shared__ int s_t[FEW_ROWS], s_x[FEW_ROWS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.n.D, R = a.n.rows, KP = D / 32, ld = 2 * D + 16;
    const int t0 = blockIdx.x * a.per, n = min(a.per, a.tiles - t0);
    const u32 slots = smem_u32(smem) + warp * (a.per * few_units(KP) * 1024);
    unsigned char* op = smem + a.per * few_units(KP) * (FEW_WARPS * 1024);
    float* red = reinterpret_cast<float*>(op + 2 * R * ld);
    u16* par = reinterpret_cast<u16*>(red + a.per * FEW_WARPS * FEW_RED);
    few_request(slots, a.w + (size_t)t0 * KP * 1024, n, KP, warp, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid == 0) dep_launch();
    few_params(a.n, par);
    const float bias = tid < n * FEW_RED ? h2f(__ldg(a.bias + (t0 + tid / FEW_RED) * 16 + (tid & 15))) : 0.f;      // of this thread's output
    __syncthreads();
    bool skip = false;
#pragma unroll 1
    for (int left = few_passes(a.first ? 1 : 2); left; left = few_passes(left - 1)) {
        const bool real = left == 1;                                               // (else the dry pass)
        const int w = few_passes(warp), l = few_passes(lane);
        if (real) dep_wait();
        if (a.first) {
            // Positions and tokens outside their ranges would index outside the tables and the caches: the step is refused. Every block
            // sees the same values. A negative position: a sequence that has not started, its row is carried along. (This kernel starts
            // when the step before is over, the later ones after it: positions do not change under them.)
            bool bad = false;
            if (tid < R) {
                const int t = __ldcg(a.t + tid * a.t_stride), x = __ldcg(a.x + tid);
                bad = t >= a.tmax || t >= a.cpos || x < 0 || x >= a.N;
                s_t[tid] = t;
                s_x[tid] = bad ? -1 : x;
            }
            if (tid == 32) bad = __ldcg(a.bar + 2) != 0u;
            skip = __syncthreads_or(bad);
            if (blockIdx.x == 0) {
                if (tid < R) a.pos[tid] = s_t[tid];
                if (tid == 0 && skip) { *a.skip = 1; atomicCAS(a.bar, 0u, 0x900u); }   // (an earlier failure keeps its own code)
            }
            few_norm<KW, WPR, FIXED, true>(a.n, true, w, l, par, op, ld, stat, [&](int row, int d) {
                const int x = s_x[row], t = max(s_t[row], 0);
                const uint2 e = __ldg(reinterpret_cast<const uint2*>(a.wte + (size_t)(x < 0 ? 0 : x) * D + d)), p = __ldg(reinterpret_cast<const uint2*>(a.wpe + (size_t)(x < 0 ? 0 : t) * D + d));
                return make_float4(h_lo(e.x) + h_lo(p.x), h_hi(e.x) + h_hi(p.x), h_lo(e.y) + h_lo(p.y), h_hi(e.y) + h_hi(p.y));
            });
        } else {
            if (tid < R) s_t[tid] = __ldcg(a.t + tid * a.t_stride);
            const void *z = real ? a.n.z : (const void*)a.w, *more = real ? a.n.more : (const void*)a.w;
            few_norm<KW, WPR, FIXED, true>(a.n, real, w, l, par, op, ld, stat, [&](int row, int d) { return State<FIXED>::load(z, more, (size_t)row * D + d); });
            skip = __ldcg(a.skip) != 0;
        }
        if (real) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        few_fold<KW>(slots, few_row(smem_u32(op), ld, R, l), n, KP, red, w, l);
        __syncthreads();
        const int o = w * 32 + l, row = (o >> 4) % FEW_ROWS, f = (t0 + o / FEW_RED) * 16 + (o & 15);
        if (row < R && o < n * FEW_RED) {
            const float v = few_sum(red, o) + bias;
            const int part = (f >= D) + (f >= 2 * D), c = f - part * D, t = s_t[row];
            if (real && part == 0) a.q[(size_t)row * D + c] = v;
            if (real && part && !skip && t >= 0) (part == 1 ? a.kc : a.vc)[row * a.seq_stride + (size_t)t * D + c] = f2h(v);
        }
    }
}

// ---- attention + projection ---------------------------------------------------------------------------------------------
struct FewAttend {
    AttArgs a;
    int rows, chunks;                 // blocks that share the positions of a sequence: rows x chunks <= 8
    const unsigned char* w;           // packed projection of the layer
    void* z;                          // the state vector that the results are added to
    static __host__ __device__ int tiles(int D) { return (D / 16 + FEW_CLUSTER - 1) / FEW_CLUSTER; }
    static __host__ __device__ int bytes(int D) { return FEW_WARPS * FEW_STAGES * 4096 + tiles(D) * 2048; }
};
// Cluster = a head, block = a sequence or a run of its positions; see pass_attend for the attention itself. 4.3 us at two sequences of 200
// positions, 4.0 at four, 5.8 at four of 900: a warp's rounds of 16 positions (0.8 us each), the cluster's exchange 0.7.
// (Two stages per warp: with four, 144 KB, the next kernel's block has no room beside it.)
template <bool FIXED>
__global__ void __launch_bounds__(FEW_THREADS) few_attend(const __grid_constant__ FewAttend a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float part[FEW_WARPS][66];
    __shared__ __align__(16) float all[FEW_CLUSTER][68];
    __shared__ __align__(16) unsigned char op[2 * FEW_ROWS * 144];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.y, c = blockIdx.x, row = c / a.chunks, chunk = c - row * a.chunks, D = a.a.D, MT = D / 16;
    const int nt = (MT - c + FEW_CLUSTER - 1) / FEW_CLUSTER;                       // tiles of 16 outputs: c, c + 8, ...
    const u32 ring = smem_u32(smem), slots = ring + FEW_WARPS * FEW_STAGES * 4096;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");          // (waited for before the other blocks' memory is written)
    for (int i = warp; i < nt; i += FEW_WARPS)
#pragma unroll
        for (int k = 0; k < 4; k++) cp16(slots + (i * 4 + k) * 512 + lane * 16, a.w + (((size_t)h * MT + c + i * FEW_CLUSTER) * 4 + k) * 512 + lane * 16);
    if (tid == 0) dep_launch();
    const bool live = row < a.rows;
    AttRow<FEW_STAGES> r(a.a, live ? row : 0, h, (chunk * FEW_WARPS + warp) * ATT_RUN, a.chunks * FEW_WARPS * ATT_RUN, ring + warp * (FEW_STAGES * 4096));
    if (live) r.request_first();
#pragma unroll 1
    for (int left = few_passes(2); left; left = few_passes(left - 1)) {
        const bool real = left == 1;
        if (real) dep_wait();
        if (live) r.run(real, part[warp]);
        __syncthreads();
        if (!real) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (live) {
            // the warps' results, merged, to all blocks of the head: warp w writes to block w
            float M = -3.0e38f, dd = 0.f, x = 0.f, y = 0.f;
#pragma unroll
            for (int i = 0; i < FEW_WARPS; i++) M = fmaxf(M, part[i][64]);
#pragma unroll
            for (int i = 0; i < FEW_WARPS; i++) { const float e = fast_exp(part[i][64] - M); dd += part[i][65] * e; x += part[i][2 * lane] * e; y += part[i][2 * lane + 1] * e; }
            const u32 to = of_block(smem_u32(&all[c][0]), warp);
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" :: "r"(to + lane * 8), "f"(x), "f"(y) : "memory");
            if (lane == 0) asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" :: "r"(to + 256), "f"(M), "f"(dd) : "memory");
        }
        cluster_sync();
        if (warp < a.rows) {
            // the runs of a sequence, merged: its head's outputs 2 lane and 2 lane + 1 into the operand
            float m[FEW_CLUSTER], M = -3.0e38f, dd = 0.f, x = 0.f, y = 0.f;
#pragma unroll
            for (int i = 0; i < FEW_CLUSTER; i++) { m[i] = i < a.chunks ? all[warp * a.chunks + i][64] : -3.0e38f; M = fmaxf(M, m[i]); }
#pragma unroll
            for (int i = 0; i < FEW_CLUSTER; i++)
                if (i < a.chunks) {
                    const float* p = all[warp * a.chunks + i];
                    const float e = fast_exp(m[i] - M);
                    dd += p[65] * e; x += p[2 * lane] * e; y += p[2 * lane + 1] * e;
                }
            const float u = dd > 0.f ? __fdividef(x, dd) : 0.f, v = dd > 0.f ? __fdividef(y, dd) : 0.f;   // (a sequence that has not started attends to nothing)
            const u32 hi = pack_h2(u, v);
            unsigned char* to = op + 2 * warp * 144 + lane * 4;
            *reinterpret_cast<u32*>(to) = hi;
            *reinterpret_cast<u32*>(to + 144) = pack_h2(u - h_lo(hi), v - h_hi(hi));
        }
        __syncthreads();
        if (real) asm volatile("cp.async.wait_all;" ::: "memory");
        u32 f[2][4];
        const u32 a_at = few_row(smem_u32(op), 144, a.rows, lane);
        ldsm4(f[0], a_at);
        ldsm4(f[1], a_at + 64);
#pragma unroll 1
        for (int i = warp; i < nt; i += FEW_WARPS) {
            float c0[2][4] = {};
            uint4 u[4];
#pragma unroll
            for (int k = 0; k < 4; k++) u[k] = lds16(slots + (i * 4 + k) * 512 + lane * 16);
#pragma unroll
            for (int k = 0; k < 2; k++) { few_mma(c0[0], u[2 * k], f[k][0], f[k][1]); few_mma(c0[1], u[2 * k + 1], f[k][2], f[k][3]); }
            if (real) few_add<FIXED>(a.z, D, a.rows, c + i * FEW_CLUSTER, c0, lane);
        }
    }
}

// ---- norm + FC + GELU + MLP projection ------------------------------------------------------------------------------------
// Two tiles of 16 features per block at an MLP width of 3,072: 96 blocks; all of a block's weights (98 KB) fit beside the attention's block on an SM.
// 4.1 us at two sequences, 4.4 at four; the reductions of 96 blocks into the same rows are much of it.
struct FewMlp {
    FewNorm n;
    const unsigned char *fc, *p2;     // packed, of the layer
    const u16* bias;
    int tiles, per;                   // tiles of 16 features, tiles per block
    float a2, k1, k2;                 // gelu_tanh
    static __host__ __device__ int bytes(int D, int rows, int per) {
        return per * ((D / 32 + 7) / 8) * 8192 + per * ((D / 16 + 7) / 8) * 4096 + 2 * rows * (2 * D + 16) + per * FEW_WARPS * FEW_RED * 4 + 2 * FEW_ROWS * (FEW_TILES * 32 + 16) + FewNorm::bytes(D);
    }
};
template <int KW, int WPR, bool FIXED>
__global__ void __launch_bounds__(FEW_THREADS, 2) few_mlp(const __grid_constant__ FewMlp a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float2 stat[FEW_WARPS];
    constexpr int ld2 = FEW_TILES * 32 + 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.n.D, R = a.n.rows, KP = D / 32, MT = D / 16, ld = 2 * D + 16;
    const int t0 = blockIdx.x * a.per, n = min(a.per, a.tiles - t0);
    // A warp's part of shared memory: its units of fc, then those of p2 (its output tiles, every eighth, x FEW_TILES tiles of the fold)
    const int fcu = 2 * a.per * few_units(KP), p2u = a.per * ((MT + FEW_WARPS - 1) / FEW_WARPS), cnt = (MT - warp + FEW_WARPS - 1) / FEW_WARPS;
    const u32 slots = smem_u32(smem) + warp * ((fcu + p2u) * 512);
    unsigned char* op = smem + (fcu + p2u) * (FEW_WARPS * 512);
    unsigned char* op2 = op + 2 * R * ld;
    float* red = reinterpret_cast<float*>(op2 + 2 * FEW_ROWS * ld2);
    u16* par = reinterpret_cast<u16*>(red + a.per * FEW_WARPS * FEW_RED);
    few_request(slots, a.fc + (size_t)t0 * KP * 1024, n, KP, warp, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 1
    for (int k = 0; k < n; k++)
#pragma unroll 1
        for (int m = 0; m < cnt; m++) cp16(slots + (fcu + m * a.per + k) * 512 + lane * 16, a.p2 + ((size_t)(t0 + k) * MT + warp + m * FEW_WARPS) * 512 + lane * 16);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid == 0) dep_launch();
    few_params(a.n, par);
    const float bias = tid < n * FEW_RED ? h2f(__ldg(a.bias + (t0 + tid / FEW_RED) * 16 + (tid & 15))) : 0.f;
    __syncthreads();
#pragma unroll 1
    for (int left = few_passes(2); left; left = few_passes(left - 1)) {
        const bool real = left == 1;
        const int w = few_passes(warp), l = few_passes(lane);
        if (real) dep_wait();
        const void* z = real ? a.n.z : (const void*)a.fc;
        few_norm<KW, WPR, FIXED, false>(a.n, real, w, l, par, op, ld, stat, [&](int row, int d) { return State<FIXED>::load(z, (size_t)row * D + d); });
        if (real) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        few_fold<KW>(slots, few_row(smem_u32(op), ld, R, l), n, KP, red, w, l);
        __syncthreads();
        const int o = w * 32 + l, row = (o >> 4) % FEW_ROWS;
        if (row < R && o < n * FEW_RED) {
            const float v = gelu_tanh(few_sum(red, o) + bias, a.a2, a.k1, a.k2);
            const u16 hi = f2h(v);
            unsigned char* to = op2 + 2 * row * ld2 + ((o / FEW_RED) * 16 + (o & 15)) * 2;
            *reinterpret_cast<u16*>(to) = hi;
            *reinterpret_cast<u16*>(to + ld2) = f2h(v - h2f(hi));
        }
        __syncthreads();
        // (every block begins with other outputs: all of them adding to the same lines at once took longer)
        u32 f[4];
        const u32 at0 = slots + fcu * 512 + l * 16;
        ldsm4(f, few_row(smem_u32(op2), ld2, R, l));
        int at = cnt ? blockIdx.x % cnt : 0;
#pragma unroll 2
        for (int x = 0; x < cnt; x++) {
            float c[2][4] = {};
            const uint4 u = lds16(at0 + at * (a.per * 512)), v = lds16(at0 + (at * a.per + n - 1) * 512);
            few_mma(c[0], u, f[0], f[1]);
            if (n > 1) few_mma(c[1], v, f[2], f[3]);
            if (real) few_add<FIXED>(a.n.into, D, R, w + at * FEW_WARPS, c, l);
            at = at + 1 == cnt ? 0 : at + 1;
        }
    }
}

}  // namespace vesta_pass
