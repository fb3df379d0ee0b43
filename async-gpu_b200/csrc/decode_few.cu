// Decode steps of few sequences as ONE persistent kernel: GPT-2 blocks, LM head, greedy pick and the next step's
// embedding, for as many steps as the launch is given.
//
// A step of one to four sequences moves every weight once and computes next to nothing; launched per operation it is a
// chain of five dependent kernels per transformer block, each a hand-over of several microseconds (GPT-2 XL, one
// sequence: 1.27 ms a step against 0.12 ms of weight bytes).  Here a cooperative grid (one block per SM) walks the whole
// depth, and a hand-over is a word:
//
//   * Every exchanged value is a 32-bit word that carries its own readiness: words are all ones (a NaN that no
//     arithmetic makes) until the producer stores the value, and the consumer polls the value itself.  No counter, no
//     fence and no barrier lies between a sum and the blocks that read it: one store and one load through L2.
//   * Words are used again every RING layers.  Whoever publishes a word returns the one of the layer after next to all
//     ones.  What lies between the uses of a word (and between a cached row and the steps that read it) is ordered by one
//     counter: in the middle of a layer one thread of every block fences and adds to it, and in the middle of the next one
//     the same thread looks, while the block waits for words anyway, whether every block has, and fences.  That covers
//     everything a block did up to the middle of the layer before last, both what it wrote and what it had read.
//   * The residual rows live in the registers of every block (a thread holds four columns); every block adds the
//     projections' words to its own copy and normalises it itself.
//   * Weights never depend on activations: one warp streams the block's part of them through a ring of tensor copies, in
//     the order in which it is used, across phases, layers and steps.  HBM is busy while words travel.
//
// Products: 16 output features x a run of K are a chunk (one tensor copy, one warp).  f32 weights multiply with FMAs.  int4
// weights stay bytes: the nibbles are the unsigned bytes of mma.sync m16n8k32, the activations its signed columns, each
// f32 value as four balanced base-256 digits of a 30-bit integer scaled by the largest of its 64 neighbours.  The integer
// sums are exact, so a product usually loses less than a chain of f32 FMAs (every input is off by 2^-30 of that largest one at
// most, which is more than an f32's own rounding for inputs below 2^-6 of it: a feature whose weights are zero where the large
// inputs are sees that), and a weight costs three instructions per eight.  An infinity makes the products of its 64 NaN.
// Group scales multiply the sums of 64 inputs in f32.
//
// What bounds a step: five hand-overs per layer of 0.9 us (a store and a load through L2 and a barrier, measured alone;
// 1.6 us with a counter), and the chain of a block's own reductions between them: LayerNorm, products, sums over warps.
// The weight bytes are hidden under that.  Steps after a prompt of 64, one / two / four sequences, us: GPT-2 Small f32 321 /
// 349 / 582 launched per operation, 192 / 232 / 307 here; GPT-2 Small int4 212 / 264, here 167 / 182; GPT-2 XL int4
// 1230 / 1635, here 976 / 1322.  At contexts of 1000 (three or two splits of a head, several turns of rows a block): Small f32 332 /
// 379 / 621, here 221 / 289 / 396.  More rows: the tensor-core GEMMs take over (their activations are fp16).
//
// Every wait is bounded: when one runs out the block records a code in the device error word, marks the session's exchanged
// words as broken (what was published and not taken back would pass for later values), waits for nothing more and leaves;
// the mark ends the other blocks' waits too.  A launch that finds it reports E_BROKEN and touches nothing, until a prompt or a
// rewind starts the words over.  Errors that other kernels of the context have left in its error word end nothing here.
//
// Replaces the per-operation launch structure of Gpt2Model::forward_cached / generate (crates/core/gpu-host/src/nn/
// models/gpt2.rs:249-288, 712-783, 1284-1339) for decode steps of few rows.
#include <cuda.h>

#include <algorithm>

#include "device_utils.cuh"
#include "model.h"
#include "tc_ptx.cuh"

namespace few {

constexpr int WARPS = 15, CT = 32 * WARPS, THREADS = CT + 32; // compute warps; one more streams the weights
constexpr int COLS = 4;          // columns of the residual rows per thread
constexpr int RING = 4;          // layers of exchange words
constexpr int MAX_SPLITS = 4;    // context splits of a head (K splits of a projection: 3)
constexpr int ATT_ROWS = 120;    // cached rows of a head that a block has in flight at a time
constexpr uint32_t EMPTY = 0xffffffffu;
enum : uint32_t { E_WAIT = 0x301, E_FULL, E_FREE, E_BROKEN };
constexpr uint32_t BROKEN = 1;   // of the session's state: a launch has given up (anything else: none has)
enum { QKV = 0, OUT = 1, FC = 2, FP = 3, HEAD = 4, MATS = 5 };
constexpr int UNIT_K[2] = {32, 64}; // inputs of a unit of K: f32, int4

struct Mat {
    int N, tiles;        // features; tiles of 16
    int splits, ku;      // parts of K (each a contribution of its own), units per part
    int cpi, kc;         // chunks of a tile's part, units of a chunk
    int bytes;           // of a chunk in shared memory
};
struct LayerPtrs {
    const float *bias[4];
    const float *ln[4]; // scale and shift of the first, scale and shift of the second LayerNorm
};
struct Params {
    Mat mat[MATS];
    const LayerPtrs *layers;
    const CUtensorMap *maps; // [layer][product]{weight, group scales}, then the output matrix's
    const float *lnf_g, *lnf_b, *wte, *wpe;
    __half *kc, *vc;    // caches [layer][seq][head][cap][64]
    size_t kv_layer;    // halves of a layer
    int n_layer, M, d, H, cap, vocab, n_positions, act, group_kb;
    float eps;
    uint32_t *tok, *history;
    int hist_cap;
    int *counters;      // {position, step}
    float *logits;      // null: not stored
    int keep_last;
    uint32_t *words;    // RING layers of slot_words each, then the picks of two steps
    int slot_words, o_att, o_lse, o_out, o_fc, o_fp; // words of a layer: q/k/v at 0
    uint32_t *state;    // {ring position of the first layer, parity of the first step, BROKEN or not, `fenced` at the start}
    uint32_t *fenced;   // fences of all blocks in the middle of a layer, ever
    uint32_t *dev_err;
    long long wait_cycles;
    int fault_layer;    // test hook: block 0 publishes no q/k/v word of that layer (-1: none)
    int n_steps, att_splits;
    int slots, slot_bytes; // chunks of the weight ring
    int xs_ld;          // staged activations: bytes between digit columns (int4), floats between rows (f32)
    int max_parts;      // sums of the warps that a block keeps in one phase
};

struct Waiter {
    volatile int *abort_flag;
    uint32_t *dev_err, *broken;
    long long limit;
    __device__ bool give_up(long long &t0) const;
};
__device__ __forceinline__ uint4 look4(const uint32_t *p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint2 look2(const uint32_t *p) {
    uint2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t look1(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void put(uint32_t *p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
// Whether to stop waiting.  Called every few hundred looks.
__device__ __noinline__ bool Waiter::give_up(long long &t0) const {
    if (*abort_flag) return true;
    const long long now = clock64();
    if (!t0) t0 = now;
    if (now - t0 <= limit && look1(broken) != BROKEN) return false;
    *abort_flag = 1;
    put(broken, BROKEN);
    atomicCAS(dev_err, 0u, (uint32_t)E_WAIT);
    return true;
}
__device__ __forceinline__ void publish(uint32_t *p, float f) {
    const uint32_t u = __float_as_uint(f);
    put(p, u == EMPTY ? 0x7fffffffu : u); // a NaN stays a NaN
}
__device__ __forceinline__ void count(uint32_t *p) { asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }
__device__ __forceinline__ uint32_t most(uint4 v) { return max(max(v.x, v.y), max(v.z, v.w)); }
__device__ __forceinline__ float4 as_float4(uint4 v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
// Four words at p, at p + stride, ... (the first n <= N of them): all requested, again until every word is there.
template <int N>
__device__ __forceinline__ void take4(const Waiter &w, const uint32_t *p, int stride, int n, uint4 (&v)[N]) {
    unsigned it = 0;
    long long t0 = 0;
#pragma unroll 1
    for (;;) {
        uint32_t top = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = i < n ? look4(p + i * stride) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < N; ++i) top = max(top, most(v[i]));
        if (top != EMPTY || ((++it & 255u) == 0 && w.give_up(t0))) return;
    }
}
__device__ __forceinline__ uint32_t take1(const Waiter &w, const uint32_t *p) {
    unsigned it = 0;
    long long t0 = 0;
#pragma unroll 1
    for (;;) {
        const uint32_t u = look1(p);
        if (u != EMPTY || ((++it & 255u) == 0 && w.give_up(t0))) return u;
    }
}

// One thread of the block, which the others meet at a barrier next: `fenced` has reached `target`, and what the blocks did
// before their part of it is ordered before what this block does from that barrier on.
__device__ __forceinline__ void settled(const Waiter &w, const uint32_t *fenced, uint32_t target) {
    unsigned it = 0;
    long long t0 = 0;
#pragma unroll 1
    while ((int)(look1(fenced) - target) < 0)
        if ((++it & 255u) == 0 && w.give_up(t0)) break;
    __threadfence();
}

// Barrier of the compute warps, whose lanes may have parted (they poll word by word).
__device__ __forceinline__ void csync() {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory");
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}

// The order in which eight neighbouring columns lie wherever this kernel keeps or exchanges them: 2 6 3 7, 0 4 1 5, as
// the nibbles of a weight word come out, high ones first.  place(c): where column c lies; a thread's four are one half.
__device__ __forceinline__ int place(int c) { return (c & ~7) + ((c & 3) < 2 ? 4 : 0) + (c & 1) * 2 + ((c >> 2) & 1); }
// This thread's four of the columns c .. c+3 of a plain row (c % 8 == 0: places 0 .. 3, else 4 .. 7).
__device__ __forceinline__ float4 quad(const float *row, int c) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(row + (c & ~7))), b = __ldg(reinterpret_cast<const float4 *>(row + (c | 4)));
    return c & 4 ? make_float4(a.x, b.x, a.y, b.y) : make_float4(a.z, b.z, a.w, b.w);
}

// Four places k .. k+3 of row m of a product's input (the whole warp takes part; `on`: this lane has some).  f32: as they
// are.  int4: as digits.  The sixteen lanes of 64 columns take the power of two that brings their largest value under
// 2^29, round to integers, and store four balanced base-256 digits, each digit a column of bytes; scale[unit][row] undoes
// the power and the weights' 16.
template <bool INT4, int MT>
__device__ __forceinline__ void stage4(uint8_t *xs, int ld, float *scale, int m, int k, float4 v, bool on) {
    if constexpr (!INT4) {
        if (on) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(xs) + m * ld + k) = v;
    } else {
        uint32_t top = __float_as_uint(fabsf(v.x));
        top = max(max(top, __float_as_uint(fabsf(v.y))), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w))));
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        const int e = top >> 23; // |v| < 2^(e - 126)
        const int up = min(155 - e, 122);
        const float f = __uint_as_float((uint32_t)(up + 127) << 23);
        const uint32_t t0 = ((uint32_t)__float2int_rn(v.x * f) + 0x00808080u) ^ 0x00808080u, t1 = ((uint32_t)__float2int_rn(v.y * f) + 0x00808080u) ^ 0x00808080u;
        const uint32_t t2 = ((uint32_t)__float2int_rn(v.z * f) + 0x00808080u) ^ 0x00808080u, t3 = ((uint32_t)__float2int_rn(v.w * f) + 0x00808080u) ^ 0x00808080u;
        if (!on) return;
        uint8_t *x = xs + 4 * m * ld + k;
        const uint32_t a = __byte_perm(t0, t1, 0x5140), b = __byte_perm(t2, t3, 0x5140); // digits 0 and 1 of two values
        const uint32_t a2 = __byte_perm(t0, t1, 0x7362), b2 = __byte_perm(t2, t3, 0x7362); // digits 2 and 3
        *reinterpret_cast<uint32_t *>(x) = __byte_perm(a, b, 0x5410);
        *reinterpret_cast<uint32_t *>(x + ld) = __byte_perm(a, b, 0x7632);
        *reinterpret_cast<uint32_t *>(x + 2 * ld) = __byte_perm(a2, b2, 0x5410);
        *reinterpret_cast<uint32_t *>(x + 3 * ld) = __byte_perm(a2, b2, 0x7632);
        // (a NaN or an infinity makes its 64 columns' products NaN)
        if ((k & 63) == 0) scale[(k >> 6) * MT + m] = __int_as_float(e == 255 ? 0x7fffffff : (123 - up) << 23);
    }
}

template <bool INT4, int MT>
__global__ void __launch_bounds__(THREADS, 1) decode_few_kernel(const __grid_constant__ Params P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ int abort_flag, gone_s, ended_s, broken_s;
    __shared__ uint32_t tok_s[4];
    __shared__ int off_s[4][CT];    // word of the sum that this thread finishes in a phase (-1: none)
    __shared__ int bias_s[4][CT];   // its feature, if it adds the bias (-1: another part does)
    __shared__ int items_s[MATS], split_s[MATS]; // items of this block in a phase; the part of K they are of
    __shared__ float2 ln_s[MT][WARPS + 1]; // (the last entry: no columns)
    __shared__ float best_v[CT / 16];
    __shared__ int best_i[CT / 16];
    __shared__ float att_s[WARPS][66];
    __shared__ __align__(16) uint32_t qkv_s[3 * 64];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nblk = gridDim.x, blk = blockIdx.x;
    const int M = P.M, d = P.d, H = P.H;
    uint8_t *ring = smem_raw + ((128u - (tc::smem_u32(smem_raw) & 127u)) & 127u);
    uint8_t *xs = ring + (size_t)P.slots * P.slot_bytes;                                        // staged activations
    float *scale = reinterpret_cast<float *>(xs + (size_t)(4 * MT) * P.xs_ld);                  // [unit][row] (f32: none)
    float *red = scale + (INT4 ? (P.xs_ld / 64 * MT + 3) / 4 * 4 : 0);             // [part][row][16]
    LayerPtrs *lp = reinterpret_cast<LayerPtrs *>(red + (size_t)P.max_parts * MT * 16);
    const uint32_t full = tc::smem_u32(lp + P.n_layer), freed = full + 8 * P.slots; // barriers

    // Two products are dealt out from the other end: the output projection, away from the blocks that have just had
    // attention, and the wide MLP product, whose blocks with a tile more have fewer of the rest.
    auto first_item = [&](int g) { return g == FC || g == OUT ? nblk - 1 - blk : blk; };
    auto n_items = [&](int g) {
        const int all = P.mat[g].tiles * P.mat[g].splits, f = first_item(g);
        return f < all ? (all - f + nblk - 1) / nblk : 0;
    };
    if (tid == 0) {
        abort_flag = 0;
        broken_s = look1(P.state + 2) == BROKEN;
#pragma unroll 1
        for (int i = 0; i < P.slots; ++i) {
            tc::mbar_init(full + 8 * i, 1);
            tc::mbar_init(freed + 8 * i, 1);
        }
        tc::fence_mbar_init();
    }
    if (tid < MATS) {
        items_s[tid] = n_items(tid);
        split_s[tid] = first_item(tid) / P.mat[tid].tiles;
    }
#pragma unroll 1
    for (int i = tid; i < P.n_layer * (int)(sizeof(LayerPtrs) / 8); i += THREADS)
        reinterpret_cast<uint64_t *>(lp)[i] = reinterpret_cast<const uint64_t *>(P.layers)[i];
    if (tid < CT)
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
            const Mat &mt = P.mat[g];
            const int item = tid / (16 * MT), m = (tid >> 4) % MT, it = first_item(g) + item * nblk, split = it / mt.tiles;
            const int n = (it - split * mt.tiles) * 16 + (tid & 15);
            const bool on = item < n_items(g) && m < M && n < mt.N;
            const int at = g == QKV ? 0 : g == OUT ? P.o_out : g == FC ? P.o_fc : P.o_fp;
            off_s[g][tid] = on ? at + (split * M + m) * mt.N + place(n) : -1;
            bias_s[g][tid] = on && split == 0 ? n : -1;
        }
    __syncthreads();
    if (broken_s) { // (by an earlier launch, or before this block had begun)
        if (tid == 0) atomicCAS(P.dev_err, 0u, (uint32_t)E_BROKEN);
        return;
    }

    const int pos0 = P.counters[0], step0 = P.counters[1];
    if (warp == WARPS) {
        // ---- one lane streams the weights: what comes next is the same in every step ----
        if (lane == 0) {
            int s = 0, n = 0;
            uint32_t ph = 1;
            bool ok = true;
#pragma unroll 1
            for (int step = 0; step < P.n_steps && ok; ++step)
#pragma unroll 1
                for (int l = 0; l < P.n_layer && ok; ++l) {
                    const CUtensorMap *mp = P.maps + (size_t)l * 8;
                    // LayerNorm vectors and biases of the layer after this one -> L2, one array by each of eight blocks
                    if (blk < 8) {
                        const LayerPtrs &nx = lp[l + 1 < P.n_layer ? l + 1 : 0];
                        const float *v = blk < 4 ? nx.ln[blk] : nx.bias[blk - 4];
                        if (v) tc::bulk_prefetch_l2(v, (uint32_t)(blk < 4 ? d : P.mat[blk - 4].N) * 4u);
                    }
#pragma unroll 1
                    for (int i = 0; i < (l + 1 < P.n_layer ? 8 : 2); i += INT4 ? 1 : 2) tc::prefetch_tmap(mp + 8 + i); // the next layer's, or the output matrix's
#pragma unroll 1
                    for (int g = 0; g < (l + 1 == P.n_layer ? 5 : 4) && ok; ++g) {
                        const Mat &mt = P.mat[g];
                        const int all = mt.tiles * mt.splits;
#pragma unroll 1
                        for (int it = first_item(g); it < all && ok; it += nblk) {
                            const int split = it / mt.tiles, tile = it - split * mt.tiles;
#pragma unroll 1
                            for (int c = 0; c < mt.cpi; ++c) {
                                const int u = split * mt.ku + c * mt.kc; // first unit of K
                                if (n >= P.slots) {
                                    ok = tc::mbar_wait1(freed + 8 * s, ph, &abort_flag, P.dev_err, E_FREE);
                                    if (!ok) break;
                                }
                                const uint32_t dst = tc::smem_u32(ring + (size_t)s * P.slot_bytes), bar = full + 8 * s;
                                tc::mbar_expect_tx(bar, mt.bytes);
                                if constexpr (INT4) {
                                    const int kb = (tile >> 3) * (mt.splits * mt.ku) + u;
                                    tc::tma_load_2d(dst, mp + 2 * g, (tile & 7) * 256, kb * 2, bar);
                                    tc::tma_load_2d(dst + mt.kc * 512, mp + 2 * g + 1, tile * 16, u / P.group_kb, bar);
                                } else {
                                    tc::tma_load_2d(dst, mp + 2 * g, tile * 16, u * 32, bar);
                                }
                                ++n;
                                if (++s == P.slots) {
                                    s = 0;
                                    ph ^= 1;
                                }
                            }
                        }
                    }
                }
            // the last filling of every slot lands before the block's memory is released, also if the other warps gave up
#pragma unroll 1
            for (int i = min(n, P.slots); i > 0; --i) {
                if (--s < 0) {
                    s = P.slots - 1;
                    ph ^= 1;
                }
                tc::mbar_drain(full + 8 * s, ph ^ 1);
            }
        }
        return;
    }

    const Waiter wait{&abort_flag, P.dev_err, P.state + 2, P.wait_cycles};
    const uint32_t ring0 = P.state[0] % RING, par0 = P.state[1] & 1; // (EMPTY, the last of its kind, after a restart)
    uint32_t all_fenced = P.state[3]; // `fenced` when every block has passed the middle of the layer before this one
    uint32_t *picks = P.words + (size_t)RING * P.slot_words;
    const int gq = lane >> 2, tq = lane & 3;
    const int c4 = tid * COLS; // this thread's places in the residual rows
    const bool mine = c4 < d;
    float4 x[MT], gam = make_float4(0.f, 0.f, 0.f, 0.f), bet = gam;
    auto norm_params = [&](const float *g, const float *b) {
        if (mine) {
            gam = quad(g, c4);
            bet = quad(b, c4);
        }
    };
    if (tid < MT) ln_s[tid][WARPS] = make_float2(0.0f, 0.0f);
    // where this thread's q/k/v sum goes in the cache (-1: a query, or none)
    long long kv_at = -1;
    bool is_v = false;
    if (bias_s[QKV][tid] >= d) {
        const int n = bias_s[QKV][tid], m = (tid >> 4) % MT;
        is_v = n >= 2 * d;
        const int c = is_v ? n - 2 * d : n - d;
        kv_at = (((long long)m * H + (c >> 6)) * P.cap) * 64 + (c & 63);
    }

    // weights of the other half and of the difference of the means where 16 lanes' statistics are merged
    float half_w, half_c;
    {
        const int from = warp * 32 * COLS + (lane & 16) * COLS, other = from ^ (16 * COLS);
        const float na = from < d ? 16.0f * COLS : 0.0f, nb = other < d ? 16.0f * COLS : 0.0f;
        half_w = na + nb > 0.0f ? nb / (na + nb) : 0.0f;
        half_c = na * half_w;
    }
    auto part_sum = [&](const float *r, int n) { // of the first n <= WARPS parts, in order
        float f = 0.0f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i)
            if (i < n) f += r[i * MT * 16];
        return f;
    };
    int base = 0;           // ring slot and phase of the next phase's first chunk
    uint32_t base_ph = 0;
    if (tid < M) tok_s[tid] = P.tok[tid];
    csync();
    uint32_t rp = ring0; // ring position of the layer
    bool gone = false;
#pragma unroll 1
    for (int step = 0; step < P.n_steps && !gone; ++step) {
        const int pos = min(pos0 + step, P.cap - 1), ctx = pos + 1;
        const int n_split = min(P.att_splits, (ctx + ATT_ROWS - 1) / ATT_ROWS);
        const int chunk = ((ctx + n_split - 1) / n_split + 3) & ~3; // rows of a split
        // this block's (sequence, head) pair and first row (there are no more items than blocks)
        const int pair = blk % (M * H), r0 = blk / (M * H) * chunk, q_at = pair / H * 3 * d + pair % H * 64;
#pragma unroll
        for (int m = 0; m < MT; ++m) { // the step's embedding
            x[m] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m < M && mine)
                x[m] = f4_add(quad(P.wte + (size_t)min(tok_s[m], (uint32_t)(P.vocab - 1)) * d, c4), quad(P.wpe + (size_t)min(pos, P.n_positions - 1) * d, c4));
        }
        norm_params(lp[0].ln[0], lp[0].ln[1]);
#pragma unroll 1
        for (int l = 0; l < P.n_layer && !gone; ++l, rp = (rp + 1) % RING, all_fenced += nblk) {
            uint32_t *slot = P.words + (size_t)rp * P.slot_words, *later = P.words + (size_t)((rp + 2) % RING) * P.slot_words;
            const bool last = l + 1 == P.n_layer;
#pragma unroll 1
            for (int g = 0; g < (last ? 5 : 4); ++g) {
                const Mat &mt = P.mat[g];
                float bias = 0.0f;
                const int parts = min(mt.cpi, WARPS), off = g != HEAD ? off_s[g][tid] : -1;
                if (g != HEAD && bias_s[g][tid] >= 0 && lp[l].bias[g]) bias = __ldg(lp[l].bias[g] + bias_s[g][tid]);
                const int items = items_s[g];

                // OUT: words of the second half of this layer and of the first of the next one (under the wait for the attention,
                // which is the longest: in the wait for the output projection's words it cost 0.3 us a layer).  HEAD: picks,
                // the last layer's cached rows.
                if ((g == OUT || g == HEAD) && tid == CT - 1) settled(wait, P.fenced, g == OUT ? all_fenced : all_fenced + nblk);

                // ---- the product's input ----
                if (g == OUT || g == FP) {
                    if (items) {
                        const int kw = mt.ku * UNIT_K[INT4], k0 = split_s[g] * kw, n4 = kw / COLS;
                        if (g == FP) {
#pragma unroll 1
                            for (int m = 0; m < M; ++m) {
                                const uint32_t *p = slot + P.o_fc + m * 4 * d + k0;
                                uint4 v[1];
                                if (tid < n4) take4<1>(wait, p + c4, 0, 1, v);
#pragma unroll 1
                                for (int e = tid; e - lane < n4; e += CT) { // warp-uniform; the next places are requested ahead
                                    const uint4 now = v[0];
                                    uint4 ahead = make_uint4(0, 0, 0, 0);
                                    if (e + CT < n4) ahead = look4(p + (e + CT) * COLS);
                                    __syncwarp();
                                    stage4<INT4, MT>(xs, P.xs_ld, scale, m, e * COLS, e < n4 ? as_float4(now) : make_float4(0.f, 0.f, 0.f, 0.f), e < n4);
                                    v[0] = ahead;
                                    if (most(ahead) == EMPTY) take4<1>(wait, p + (e + CT) * COLS, 0, 1, v);
                                }
                            }
                        } else if (warp * 32 < n4) { // (n4 <= CT) parts of a head's context: each weighs as much as its share of the sum of exponentials
                            const bool on = tid < n4;
#pragma unroll 1
                            for (int m = 0; m < M; ++m) {
                                float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (on) {
                                    const uint32_t *p = slot + P.o_att + m * d + k0 + c4;
                                    if (n_split == 1) {
                                        uint4 v[1];
                                        take4<1>(wait, p, 0, 1, v);
                                        o = as_float4(v[0]);
                                    } else {
                                        uint4 v[MAX_SPLITS];
                                        take4<MAX_SPLITS>(wait, p, M * d, n_split, v);
                                        float lse[MAX_SPLITS], top = -INFINITY, sum = 0.0f;
#pragma unroll
                                        for (int s = 0; s < MAX_SPLITS; ++s) {
                                            lse[s] = s < n_split ? __uint_as_float(take1(wait, slot + P.o_lse + (s * M + m) * H + ((k0 + c4) >> 6))) : -INFINITY;
                                            top = fmaxf(top, lse[s]);
                                        }
#pragma unroll
                                        for (int s = 0; s < MAX_SPLITS; ++s)
                                            if (s < n_split) {
                                                const float w = exp2f(lse[s] - top);
                                                const float4 a = as_float4(v[s]);
                                                sum += w;
                                                o = make_float4(fmaf(w, a.x, o.x), fmaf(w, a.y, o.y), fmaf(w, a.z, o.z), fmaf(w, a.w, o.w));
                                            }
                                        const float inv = 1.0f / sum;
                                        o = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
                                    }
                                }
                                __syncwarp();
                                stage4<INT4, MT>(xs, P.xs_ld, scale, m, c4, o, on);
                            }
                        }
                        csync();
                    }
                } else {
                    // residual rows: add the projection's contributions, then LayerNorm.  Mean and sum of squares about it
                    // per warp, then over the warps with the distances of their means.
                    if (g != QKV || l) {
                        const uint32_t *p = g == FC ? slot + P.o_out : (g == HEAD ? slot : P.words + (size_t)((rp + RING - 1) % RING) * P.slot_words) + P.o_fp;
                        const int splits = P.mat[g == FC ? OUT : FP].splits;
                        if (mine)
#pragma unroll
                            for (int m = 0; m < MT; ++m)
                                if (m < M) {
                                    uint4 v[3];
                                    take4<3>(wait, p + m * d + c4, M * d, splits, v);
                                    x[m] = f4_add(f4_add(f4_add(x[m], as_float4(v[0])), as_float4(v[1])), as_float4(v[2]));
                                }
                    }
                    __syncwarp();
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        float mean = ((x[m].x + x[m].y) + (x[m].z + x[m].w)) * 0.25f;
                        float4 t = make_float4(x[m].x - mean, x[m].y - mean, x[m].z - mean, x[m].w - mean);
                        float q = fmaf(t.x, t.x, t.y * t.y) + fmaf(t.z, t.z, t.w * t.w); // zero past the row's end
#pragma unroll
                        for (int k = 0; k < 5; ++k) { // two halves of equal or (past the row's end) no size
                            const float dm = __shfl_xor_sync(0xffffffffu, mean, 1 << k) - mean, oq = __shfl_xor_sync(0xffffffffu, q, 1 << k);
                            mean = fmaf(dm, k < 4 ? 0.5f : half_w, mean);
                            q = fmaf(dm * dm, k < 4 ? (float)(2 << k) : half_c, q + oq);
                        }
                        if (lane == 0) ln_s[m][warp] = make_float2(mean, q);
                    }
                    if (g == QKV && tid == 0) gone_s = abort_flag;
                    csync();
                    if (g == QKV) gone = gone_s != 0;
                    const int lw = lane & 15;
                    const float nl = (float)max(0, min(32 * COLS, d - lw * 32 * COLS)), inv_d = 1.0f / (float)d;
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const float2 e = ln_s[m][lw];
                        float s = nl * e.x;
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                        const float mean = s * inv_d;
                        float q = fmaf(nl * (e.x - mean), e.x - mean, e.y);
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                        const float rs = rsqrtf(q * inv_d + P.eps);
                        stage4<INT4, MT>(xs, P.xs_ld, scale, m, c4,
                                         make_float4((x[m].x - mean) * rs * gam.x + bet.x, (x[m].y - mean) * rs * gam.y + bet.y,
                                                     (x[m].z - mean) * rs * gam.z + bet.z, (x[m].w - mean) * rs * gam.w + bet.w), mine);
                    }
                    csync();
                    if (gone) break;
                    if (g == QKV) norm_params(lp[l].ln[2], lp[l].ln[3]);
                    else if (g == FC && !last) norm_params(lp[l + 1].ln[0], lp[l + 1].ln[1]);
                    else if (g == FC) norm_params(P.lnf_g, P.lnf_b);
                }

                // ---- the block's sums, chunk by chunk, in `red` ----
                // A ring slot always belongs to the same warp (their number is a multiple of the warps'), so that nobody can ask for
                // a slot's next filling while its last one is still on its way.
                const int nc = items * mt.cpi, rot = warp - base % WARPS, first = rot < 0 ? rot + WARPS : rot;
                int kpos = first, sl = base + first;
                uint32_t sph = base_ph;
                float *dst = red;
#pragma unroll 1
                while (kpos >= mt.cpi) {
                    kpos -= mt.cpi;
                    dst += parts * MT * 16;
                }
                int kfirst = kpos;
                dst += kpos * MT * 16;
                if (sl >= P.slots) {
                    sl -= P.slots;
                    sph ^= 1;
                }
                float acc[INT4 ? 2 : MT][INT4 ? 1 : 4] = {};
#pragma unroll 1
                for (int c = first; c < nc; c += WARPS) {
                    tc::mbar_wait(full + 8 * sl, sph, &abort_flag, P.dev_err, E_FULL);
                    const uint8_t *u = ring + (size_t)sl * P.slot_bytes;
                    const int u0 = kpos * mt.kc, units = min(mt.kc, mt.ku - u0); // units of the staged input
                    if constexpr (INT4) {
                        const uint32_t *w = reinterpret_cast<const uint32_t *>(u) + gq * 4 + tq;
                        const __half *sc = reinterpret_cast<const __half *>(u + mt.kc * 512) + gq;
                        const uint8_t *xb = xs + (size_t)gq * P.xs_ld + u0 * 64 + 8 * tq;
                        const float *sx = scale + u0 * MT + (MT == 2 ? tq >> 1 : 0);
                        const bool col = MT == 2 || gq < 4;
                        int km = (split_s[g] * mt.ku + u0) % P.group_kb;
                        float t0 = acc[0][0], t1 = acc[1][0];
#pragma unroll 5
                        for (int i = 0; i < units; ++i) {
                            const uint32_t hi = 0xf0f0f0f0u, flip = 0x80808080u, w0 = w[0], w1 = w[32], w2 = w[64], w3 = w[96];
                            const uint2 b0 = col ? *reinterpret_cast<const uint2 *>(xb) : make_uint2(0, 0);
                            const uint2 b1 = col ? *reinterpret_cast<const uint2 *>(xb + 32) : make_uint2(0, 0);
                            const float s = *sx, s0 = __half2float(sc[0]) * s, s1 = __half2float(sc[8]) * s;
                            int p0[4] = {0, 0, 0, 0}, p1[4] = {0, 0, 0, 0};
                            // a nibble in the upper half of a byte, its top bit turned, is 16 (nibble - 8)
                            mma_s8(p0, (w0 & hi) ^ flip, (w1 & hi) ^ flip, ((w0 << 4) & hi) ^ flip, ((w1 << 4) & hi) ^ flip, b0);
                            mma_s8(p1, (w2 & hi) ^ flip, (w3 & hi) ^ flip, ((w2 << 4) & hi) ^ flip, ((w3 << 4) & hi) ^ flip, b1);
                            t0 = fmaf(s0, (float)((p0[0] + p1[0]) + ((p0[1] + p1[1]) << 8)), t0);
                            t1 = fmaf(s1, (float)((p0[2] + p1[2]) + ((p0[3] + p1[3]) << 8)), t1);
                            w += 128;
                            xb += 64;
                            sx += MT;
                            if (++km == P.group_kb) {
                                km = 0;
                                sc += 16;
                            }
                        }
                        acc[0][0] = t0;
                        acc[1][0] = t1;
                    } else {
                        const float4 *w = reinterpret_cast<const float4 *>(u) + lane;
                        const float *xr = reinterpret_cast<const float *>(xs) + u0 * 32 + place(gq);
#pragma unroll 2
                        for (int i = 0; i < units; ++i) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float4 wv = w[j * 32];
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    const float xv = xr[m * P.xs_ld + j * 8];
                                    acc[m][0] = fmaf(xv, wv.x, acc[m][0]);
                                    acc[m][1] = fmaf(xv, wv.y, acc[m][1]);
                                    acc[m][2] = fmaf(xv, wv.z, acc[m][2]);
                                    acc[m][3] = fmaf(xv, wv.w, acc[m][3]);
                                }
                            }
                            w += 128;
                            xr += 32;
                        }
                    }
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(freed + 8 * sl);
                    sl += WARPS;
                    if (sl >= P.slots) {
                        sl -= P.slots;
                        sph ^= 1;
                    }
                    kpos += WARPS;
                    if (kpos < mt.cpi) continue; // more of the same tile
                    if constexpr (INT4) {
                        float t0 = acc[0][0], t1 = acc[1][0];
                        if (tq & 1) { // the upper two digits
                            t0 *= 65536.0f;
                            t1 *= 65536.0f;
                        }
                        t0 += __shfl_xor_sync(0xffffffffu, t0, 1);
                        t1 += __shfl_xor_sync(0xffffffffu, t1, 1);
                        if ((tq & 1) == 0 && (tq >> 1) < MT) {
                            dst[(tq >> 1) * 16 + gq] = t0;
                            dst[(tq >> 1) * 16 + gq + 8] = t1;
                        }
                        acc[0][0] = acc[1][0] = 0.0f;
                    } else {
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                acc[m][j] += __shfl_xor_sync(0xffffffffu, acc[m][j], 4);
                                acc[m][j] += __shfl_xor_sync(0xffffffffu, acc[m][j], 8);
                                acc[m][j] += __shfl_xor_sync(0xffffffffu, acc[m][j], 16);
                            }
                            if (gq == 0) *reinterpret_cast<float4 *>(dst + m * 16 + tq * 4) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
#pragma unroll
                            for (int j = 0; j < 4; ++j) acc[m][j] = 0.0f;
                        }
                    }
                    // the warp's first chunk of its next tile
                    dst -= kfirst * MT * 16;
#pragma unroll 1
                    while (kpos >= mt.cpi) {
                        kpos -= mt.cpi;
                        dst += parts * MT * 16;
                    }
                    kfirst = kpos;
                    dst += kpos * MT * 16;
                }
                base += nc;
#pragma unroll 1
                while (base >= P.slots) {
                    base -= P.slots;
                    base_ph ^= 1;
                }
                if (!items) continue; // (uniform for the block)
                csync();

                // ---- finished sums leave ----
                if (g != HEAD) {
                    if (off >= 0) {
                        float f = part_sum(red + tid / (16 * MT) * parts * MT * 16 + (tid & (16 * MT - 1)), parts);
                        f += bias;
                        if (g == FC) f = P.act == B200NN_ACT_GELU_SIGMOID ? gelu_sigmoid_f(f) : gelu_tanh_f(f);
                        if (!(g == QKV && blk == 0 && l == P.fault_layer)) publish(slot + off, f);
                        put(later + off, EMPTY);
                        if (g == QKV && kv_at >= 0) ((is_v ? P.vc : P.kc) + (size_t)l * P.kv_layer)[kv_at + (long long)pos * 64] = __float2half_rn(f);
                    }
                    // behind the barrier: all that this block has read, its cache rows, and what it has returned to EMPTY but for
                    // this product's words, which the next layer's fence covers
                    if (g == FC && tid == CT - 1) {
                        __threadfence();
                        count(P.fenced);
                    }
                }
                if (g == QKV) {
                    // ---- attention: a (sequence, head) pair and a part of its context per block ----
                    if (blk < M * H * P.att_splits) {
                        if (tid < 64) put(later + P.o_att + blk * 64 + tid, EMPTY);
                        if (tid == 64) put(later + P.o_lse + blk, EMPTY);
                    }
                    if (blk < M * H * n_split) {
                        const int r1 = min(r0 + chunk, ctx), lg = lane >> 3, c = lane & 7;
                        const size_t at = ((size_t)l * P.kv_layer + (size_t)pair * P.cap * 64) / 8 + c;
                        const uint4 *kp = reinterpret_cast<const uint4 *>(P.kc) + at, *vp = reinterpret_cast<const uint4 *>(P.vc) + at;
                        if (tid < 2 && !last && min(r1, pos) > r0) // the next layer's cached rows -> L2 (a hint)
                            tc::bulk_prefetch_l2((tid ? vp : kp) - c + P.kv_layer / 8 + (size_t)r0 * 8, (uint32_t)(min(r1, pos) - r0) * 128u);
                        constexpr int TRIP = WARPS * 4, R = ATT_ROWS / TRIP; // rows of the block per row of a lane group; rows of a group in flight
                        uint4 kr[R], vr[R];
                        auto request = [&](int first) { // cached rows first + j * TRIP (those of earlier steps)
#pragma unroll
                            for (int j = 0; j < R; ++j) {
                                const int row = first + j * TRIP;
                                kr[j] = vr[j] = make_uint4(0, 0, 0, 0);
                                if (row < r1 && row < pos) {
                                    kr[j] = __ldcg(kp + (size_t)row * 8);
                                    vr[j] = __ldcg(vp + (size_t)row * 8);
                                }
                            }
                        };
                        request(r0 + warp * 4 + lg);
                        float q[8];
                        uint4 kn, vn; // this step's row: its words, rounded as the cache holds them
                        {
                            if (tid < 48) { // q, k and v of the head: sixteen threads each
                                uint4 one[1];
                                take4<1>(wait, slot + q_at + (tid >> 4) * d + (tid & 15) * 4, 0, 1, one);
                                *reinterpret_cast<uint4 *>(&qkv_s[tid * 4]) = one[0];
                            }
                            csync();
                            const uint4 *qs = reinterpret_cast<const uint4 *>(qkv_s) + c * 2;
                            const uint4 t[3] = {qs[0], qs[16], qs[32]}, u[3] = {qs[1], qs[17], qs[33]}; // places 0 .. 7: columns 2 6 3 7, 0 4 1 5
                            const float sc = 0.125f * 1.4426950408889634f;
                            const float4 a = as_float4(t[0]), b = as_float4(u[0]);
                            q[2] = a.x * sc; q[6] = a.y * sc; q[3] = a.z * sc; q[7] = a.w * sc;
                            q[0] = b.x * sc; q[4] = b.y * sc; q[1] = b.z * sc; q[5] = b.w * sc;
                            auto halves = [&](uint4 lo, uint4 hi) {
                                const float4 a = as_float4(lo), b = as_float4(hi);
                                return make_uint4(pack_f16x2(b.x, b.z), pack_f16x2(a.x, a.z), pack_f16x2(b.y, b.w), pack_f16x2(a.y, a.w));
                            };
                            kn = halves(t[1], u[1]);
                            vn = halves(t[2], u[2]);
                        }
                        __syncwarp();
                        float mx = -1.0e30f, sum = 0.0f, acc[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 1
                        for (int first = r0 + warp * 4; first < r1; first += ATT_ROWS) { // warp-uniform
                            if (first != r0 + warp * 4) request(first + lg);
                            float sc[R];
#pragma unroll
                            for (int j = 0; j < R; ++j)
                                if (first + lg + j * TRIP == pos) {
                                    kr[j] = kn;
                                    vr[j] = vn;
                                }
#pragma unroll
                            for (int j = 0; j < R; ++j) {
                                const __half2 *kh = reinterpret_cast<const __half2 *>(&kr[j]);
                                float t = 0.0f;
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const float2 f = __half22float2(kh[i]);
                                    t = fmaf(q[2 * i], f.x, t);
                                    t = fmaf(q[2 * i + 1], f.y, t);
                                }
                                sc[j] = t;
                            }
#pragma unroll
                            for (int o = 1; o < 8; o <<= 1)
#pragma unroll
                                for (int j = 0; j < R; ++j) sc[j] += __shfl_xor_sync(0xffffffffu, sc[j], o);
                            float top = mx;
#pragma unroll
                            for (int j = 0; j < R; ++j)
                                if (first + lg + j * TRIP < r1) top = fmaxf(top, sc[j]);
                            const float corr = exp2f(mx - top);
                            sum *= corr;
#pragma unroll
                            for (int i = 0; i < 8; ++i) acc[i] *= corr;
#pragma unroll
                            for (int j = 0; j < R; ++j) {
                                const float p = first + lg + j * TRIP < r1 ? exp2f(sc[j] - top) : 0.0f;
                                sum += p;
                                const __half2 *vh = reinterpret_cast<const __half2 *>(&vr[j]);
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const float2 f = __half22float2(vh[i]);
                                    acc[2 * i] = fmaf(p, f.x, acc[2 * i]);
                                    acc[2 * i + 1] = fmaf(p, f.y, acc[2 * i + 1]);
                                }
                            }
                            mx = top;
                        }
                        // the four lane groups, then the warps
#pragma unroll
                        for (int o = 8; o < 32; o <<= 1) {
                            const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, sum, o);
                            const float top = fmaxf(mx, om), a = exp2f(mx - top), b = exp2f(om - top);
                            sum = sum * a + os * b;
#pragma unroll
                            for (int i = 0; i < 8; ++i) acc[i] = acc[i] * a + __shfl_xor_sync(0xffffffffu, acc[i], o) * b;
                            mx = top;
                        }
                        if (lane < 8) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) att_s[warp][lane * 8 + i] = acc[i];
                            if (lane == 0) {
                                att_s[warp][64] = mx;
                                att_s[warp][65] = sum;
                            }
                        }
                        csync();
                        if (tid < 64) {
                            const int w = lane & 15;
                            const float wm = w < WARPS ? att_s[w][64] : -1.0e30f;
                            float top = wm;
#pragma unroll
                            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                            const float e = w < WARPS ? exp2f(wm - top) : 0.0f;
                            float t = w < WARPS ? e * att_s[w][65] : 0.0f, o = 0.0f;
#pragma unroll
                            for (int s = 8; s > 0; s >>= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
#pragma unroll
                            for (int s = 0; s < WARPS; ++s) o = fmaf(__shfl_sync(0xffffffffu, e, s), att_s[s][tid], o);
                            publish(slot + P.o_att + blk * 64 + place(tid), o / t);
                            if (n_split > 1 && tid == 0) publish(slot + P.o_lse + blk, top + log2f(t));
                        }
                    }
                }
            }
            if (gone) break;
        }
        if (gone) break;

        // ---- greedy pick ----
        {
            const int m = (tid >> 4) % MT, items = items_s[HEAD], cpi = P.mat[HEAD].cpi;
            float bv = -INFINITY;
            int bi = P.keep_last ? -1 : 0x7fffffff;
            constexpr int ALL = CT / (16 * MT) * (16 * MT); // threads that keep to one row
#pragma unroll 1
            for (int v = tid < ALL ? tid : items * 16 * MT; v < items * 16 * MT; v += ALL) {
                const int item = v / (16 * MT), n = (blk + item * nblk) * 16 + (v & 15);
                if (m >= M || n >= P.vocab) continue;
                const float f = part_sum(red + item * min(cpi, WARPS) * MT * 16 + (v & (16 * MT - 1)), min(cpi, WARPS));
                if (P.logits) P.logits[(size_t)m * P.vocab + n] = f;
                amax_merge(bv, bi, f, n, P.keep_last);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                amax_merge(bv, bi, ov, oi, P.keep_last);
            }
            if ((lane & 15) == 0) {
                best_v[tid >> 4] = bv;
                best_i[tid >> 4] = bi;
            }
        }
        csync();
        uint32_t *pick = picks + (size_t)((par0 + step) & 1) * nblk * MT * 2;
        if (warp == 0) {
            float bv = lane < CT / 16 ? best_v[lane] : -INFINITY;
            int bi = lane < CT / 16 ? best_i[lane] : P.keep_last ? -1 : 0x7fffffff;
#pragma unroll
            for (int o = 16; o >= MT; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                amax_merge(bv, bi, ov, oi, P.keep_last);
            }
            if (lane < MT) {
                publish(pick + (size_t)(blk * MT + lane) * 2, bv);
                put(pick + (size_t)(blk * MT + lane) * 2 + 1, (uint32_t)bi + 2u); // -1 .. 0x7fffffff: never EMPTY
            }
        }
        if (warp < M) { // a warp per row over all blocks' candidates
            float bv = -INFINITY;
            int bi = P.keep_last ? -1 : 0x7fffffff;
#pragma unroll 1
            for (int b = lane; b < nblk; b += 32) {
                const uint32_t *p = pick + (size_t)(b * MT + warp) * 2;
                uint2 u = look2(p);
                unsigned it = 0;
                long long t0 = 0;
#pragma unroll 1
                while (u.x == EMPTY || u.y == EMPTY) {
                    u = look2(p);
                    if ((++it & 255u) == 0 && wait.give_up(t0)) break;
                }
                amax_merge(bv, bi, __uint_as_float(u.x), (int)(u.y - 2u), P.keep_last);
            }
            __syncwarp();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                amax_merge(bv, bi, ov, oi, P.keep_last);
            }
            if (lane == 0) tok_s[warp] = bi < 0 || bi >= P.vocab ? 0u : (uint32_t)bi;
        }
        csync();
        if (tid == 0) ended_s = abort_flag || (blk == 0 && step + 1 == P.n_steps && look1(P.state + 2) == BROKEN);
        csync();
        gone = ended_s != 0; // nothing of a step that was given up is stored
        if (gone) break;
        // those of the step before have been read: every block has fenced in this step's last layer
        if (tid < 2 * MT) put(picks + (size_t)((par0 + step + 1) & 1) * nblk * MT * 2 + (size_t)blk * MT * 2 + tid, EMPTY);
        if (blk == 0 && tid < M && step0 + step < P.hist_cap) P.history[(size_t)tid * P.hist_cap + step0 + step] = tok_s[tid];
    }
    if (gone) {
        if (tid == 0) put(P.state + 2, BROKEN); // (a copy that did not come ends a block too)
    } else if (blk == 0) { // every block has read these: it has published since
        if (tid < M) P.tok[tid] = tok_s[tid];
        if (tid == 0) {
            P.counters[0] = pos0 + P.n_steps;
            P.counters[1] = step0 + P.n_steps;
            P.state[0] = rp;
            P.state[1] = (par0 + P.n_steps) & 1;
            P.state[3] = all_fenced;
        }
    }
}

// What a launch needs, worked out from the model's shapes.
struct Plan {
    int grid = 0, MT = 0, xs_ld = 0, att_splits = 0, slots = 0, slot_bytes = 0, max_parts = 0;
    Mat mat[MATS];
    size_t smem = 0, slot_words = 0, o_att = 0, o_lse = 0, o_out = 0, o_fc = 0, o_fp = 0, words = 0;
};
constexpr size_t SMEM_MAX = 206 * 1024; // dynamic; the kernel's tables take some of the rest

static bool make_plan(const b200nn_gpt2 *m, int M, int cap, Plan *out) {
    const b200nn_ctx *ctx = m->ctx;
    const int d = m->cfg.n_embd, H = m->cfg.n_head, L = m->cfg.n_layer;
    const bool int4 = m->int4;
    Plan p;
    p.MT = M <= 1 ? 1 : M <= 2 ? 2 : 4;
    if (M < 1 || M > (int4 ? 2 : 4) || M * H > std::min(ctx->sm_count, 3 * d / 16) || d % 64 != 0 || d > CT * COLS || L < 1 || !ctx->encode_tiled) return false;
    const int unit_k = UNIT_K[int4], gkb = int4 ? m->blocks[0].qkv.q.group / 64 : 1;
    const LinearAny *lin[MATS] = {&m->blocks[0].qkv, &m->blocks[0].proj, &m->blocks[0].fc, &m->blocks[0].fcproj, &m->lm_head};
    auto fits = [&](const LinearAny &l, const LinearAny &like) {
        if (l.int4 != int4 || l.b16 || l.K != like.K || l.N != like.N || l.K % unit_k != 0) return false;
        if (int4) return l.q.fast && l.q.group == m->blocks[0].qkv.q.group && l.q.group % 64 == 0;
        return l.f.ld() % 4 == 0 && ((uintptr_t)l.f.w_kn->p & 15) == 0;
    };
    for (int g = 0; g < MATS; ++g) {
        if (!fits(*lin[g], *lin[g])) return false;
        p.mat[g].N = lin[g]->N;
        p.mat[g].tiles = (lin[g]->N + 15) / 16;
        p.mat[g].splits = 1;
        p.mat[g].ku = lin[g]->K / unit_k;
    }
    for (const BlockW &b : m->blocks)
        if (!fits(b.qkv, *lin[QKV]) || !fits(b.proj, *lin[OUT]) || !fits(b.fc, *lin[FC]) || !fits(b.fcproj, *lin[FP])) return false;
    // every block owns a tile of the q/k/v product and of the wide MLP product, in which it counts itself past the middle of a layer
    p.grid = std::min(ctx->sm_count, p.mat[QKV].tiles);
    if (p.mat[FC].tiles < p.grid) return false;
    // the projections back to the model width have few tiles: their K is split where that gives idle blocks work
    for (int g : {OUT, FP})
        for (int s = std::min(3, p.grid / p.mat[g].tiles); s > 1; --s)
            if (p.mat[g].ku % s == 0 && (p.mat[g].ku / s * unit_k) % 64 == 0) {
                p.mat[g].splits = s;
                p.mat[g].ku /= s;
                break;
            }
    int kmax = 0;
    for (int g = 0; g < MATS; ++g) {
        Mat &t = p.mat[g];
        const int items = (t.tiles * t.splits + p.grid - 1) / p.grid;
        if (g != HEAD && items * 16 * p.MT > CT) return false;
        // a chunk is one warp's work: as many units as keep the busiest warp's share small (a chunk costs about one more)
        const int most = int4 ? 7 : 3;
        int best = 1 << 30;
        for (int kc = 1; kc <= std::min(most, t.ku); ++kc) {
            const int cpi = (t.ku + kc - 1) / kc, cost = (items * cpi + WARPS - 1) / WARPS * (kc + 1);
            if (cost < best || (cost == best && cpi < t.cpi)) {
                best = cost;
                t.kc = kc;
                t.cpi = cpi;
            }
        }
        t.bytes = int4 ? t.kc * 512 + ((t.kc - 1) / gkb + 2) * 32 : t.kc * 2048;
        p.slot_bytes = std::max(p.slot_bytes, (t.bytes + 127) & ~127);
        p.max_parts = std::max(p.max_parts, items * std::min(t.cpi, WARPS));
        kmax = std::max(kmax, t.ku * unit_k);
    }
    // int4: digit columns 32 bytes apart modulo 128, so that the four columns of a half warp read different banks
    p.xs_ld = int4 ? (kmax + 127) / 128 * 128 + 32 : kmax;
    const size_t rest = 128 + (size_t)4 * p.MT * p.xs_ld + (int4 ? (size_t)(p.xs_ld / 64 * p.MT + 3) / 4 * 16 : 0) + (size_t)p.max_parts * p.MT * 64 +
                        (size_t)L * sizeof(LayerPtrs);
    if (rest >= SMEM_MAX) return false;
    p.slots = (int)std::min<size_t>(6, (SMEM_MAX - rest) / ((size_t)p.slot_bytes + 16) / WARPS) * WARPS;
    if (!p.slots) return false;
    p.smem = rest + (size_t)p.slots * (p.slot_bytes + 16);
    p.att_splits = std::max(1, std::min({MAX_SPLITS, p.grid / std::max(1, M * H), (cap + ATT_ROWS - 1) / ATT_ROWS}));
    size_t o = (size_t)M * 3 * d;
    p.o_att = o;
    o += (size_t)p.att_splits * M * H * 64;
    p.o_lse = o;
    o += ((size_t)p.att_splits * M * H + 3) & ~(size_t)3;
    p.o_out = o;
    o += (size_t)p.mat[OUT].splits * M * d;
    p.o_fc = o;
    o += (size_t)M * 4 * d;
    p.o_fp = o;
    o += (size_t)p.mat[FP].splits * M * d;
    p.slot_words = (o + 31) & ~(size_t)31;
    p.words = RING * p.slot_words + (size_t)2 * p.grid * p.MT * 2;
    *out = p;
    return true;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static int encode2d(b200nn_ctx *ctx, CUtensorMap *map, CUtensorMapDataType type, void *p, size_t x, size_t y, size_t row_bytes, int bx, int by) {
    const cuuint64_t dim[2] = {x, y}, stride[1] = {row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)bx, (cuuint32_t)by}, one[2] = {1, 1};
    const CUresult r = ((EncodeTiledFn)ctx->encode_tiled)(map, type, 2, p, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(ctx, B200NN_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return B200NN_OK;
}
// {weight, group scales} of one product.  The packed tiles as rows of 2048 bytes, a plane of a K block each: sixteen
// features are 256 bytes of every row.
static int encode_mat(b200nn_ctx *ctx, const LinearAny &l, const Mat &t, CUtensorMap *map) {
    if (!l.int4) return encode2d(ctx, map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, l.f.w_kn->p, l.N, l.K, (size_t)l.f.ld() * 4, 16, t.kc * 32);
    TRY(encode2d(ctx, map, CU_TENSOR_MAP_DATA_TYPE_UINT8, l.q.tiled->p, 2048, (size_t)l.q.n_tiles * l.q.k_blocks * 2, 2048, 256, 2 * t.kc));
    return encode2d(ctx, map + 1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, l.q.scales_h->p, l.q.n_pad, l.q.n_groups, (size_t)l.q.n_pad * 2, 16,
                    (t.kc - 1) / (l.q.group / 64) + 2);
}

using Kernel = void (*)(const Params);
static Kernel kernel_of(bool int4, int MT) {
    if (int4) return MT == 1 ? decode_few_kernel<true, 1> : decode_few_kernel<true, 2>;
    return MT == 1 ? decode_few_kernel<false, 1> : MT == 2 ? decode_few_kernel<false, 2> : decode_few_kernel<false, 4>;
}

}  // namespace few

// Sessions whose steps can run this way: see make_plan; the rest keep one kernel per operation.
bool decode_few_supported(const b200nn_gpt2 *m, int rows, int cap) {
    few::Plan p;
    b200nn_ctx *ctx = m->ctx;
    if (model_act_half(m, rows) || !few::make_plan(m, rows, cap, &p)) return false;
    int coop = 0, per_sm = 0;
    const few::Kernel k = few::kernel_of(m->int4, p.MT);
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, few::SMEM_MAX) != cudaSuccess) {
        cudaGetLastError(); // (launches look at the last error)
        return false;
    }
    prefer_max_smem(k);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, few::THREADS, p.smem) != cudaSuccess) cudaGetLastError();
    return coop && per_sm * ctx->sm_count >= p.grid;
}

// Whether the steps are faster this way.  A layer gains up to 40 us here (int4 of 512 to 1600 columns: 3 to 10), a launch costs 20
// to 25 us more than a graph's, and the output matrix has fewer blocks (those of the q/k/v product) and one read of its
// weights for them all.  Steps taken and read one by one, us, here / one kernel per operation, 50257 tokens: width 64, 2 layers
// int4 150 / 49, f32 116 / 50; 256, 4 layers 88 / 79, 106 / 87; 512, 8 layers 125 / 145, 163 / 188; 1024 int4, 6 layers 148 / 143; 1920 int4, 8
// layers 286 / 275, f32 460 / 679.  In runs of 32 steps: 118 / 37, 89 / 37; 58 / 68, 84 / 76; 99 / 131, 136 / 177; 118 / 130; 255 / 264, 438 / 666.
// Below 512 columns a layer gains little or (several sequences, long contexts) nothing.  A larger vocabulary asks for as many
// more layers.
bool decode_few_pays(const b200nn_gpt2 *m) {
    const int d = m->cfg.n_embd, need = m->int4 && (d < 640 || d > 1600) ? 12 : 6;
    return d >= 512 && (long long)m->cfg.n_layer * 65536 >= (long long)need * std::max(65536, (int)m->cfg.vocab_size);
}

// Steps of a launch.  The kernel holds every SM until it ends, and other streams wait for it: about 5 ms, by the 10 to 30 us
// (int4, growing with the width) and 12 to 60 us (f32) that a layer was measured at.
int decode_few_steps(const b200nn_gpt2 *m) {
    const int layer_us = std::max(15, m->cfg.n_embd / (m->int4 ? 70 : 32));
    return std::max(1, std::min(32, 5000 / (layer_us * m->cfg.n_layer)));
}

// All words EMPTY (the ring's position, the parity and the counter too: any are as good; not BROKEN): before the first step after a
// prompt or a rewind.
int decode_few_restart(b200nn_session *s) {
    CK(s->m->ctx, cudaMemsetAsync(s->few_words->p, 0xff, s->few_words->bytes, s->m->ctx->stream));
    return B200NN_OK;
}

int decode_few_prepare(b200nn_session *s) {
    b200nn_gpt2 *m = s->gpt2;
    b200nn_ctx *ctx = m->ctx;
    few::Plan p;
    if (!few::make_plan(m, (int)s->batch, (int)s->kv.cap, &p)) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "decode_few: no plan");
    TRY(dev_alloc(ctx, p.words * 4 + 256, &s->few_words));
    s->few_broken = (const uint32_t *)s->few_words->p + p.words + 2;
    TRY(decode_few_restart(s));
    if (m->few_maps) return B200NN_OK; // the chunks' shapes depend on the model alone
    const size_t L = m->cfg.n_layer;
    std::vector<few::LayerPtrs> h(L);
    std::vector<CUtensorMap> maps(8 * L + 2);
    for (size_t l = 0; l < L; ++l) {
        const BlockW &b = m->blocks[l];
        const LinearAny *lin[4] = {&b.qkv, &b.proj, &b.fc, &b.fcproj};
        const std::shared_ptr<DevBuf> *ln[4] = {&b.ln1_g, &b.ln1_b, &b.ln2_g, &b.ln2_b};
        for (int g = 0; g < 4; ++g) {
            h[l].bias[g] = lin[g]->bias();
            h[l].ln[g] = (const float *)(*ln[g])->p;
            TRY(few::encode_mat(ctx, *lin[g], p.mat[g], &maps[8 * l + 2 * g]));
        }
    }
    TRY(few::encode_mat(ctx, m->lm_head, p.mat[few::HEAD], &maps[8 * L]));
    std::shared_ptr<DevBuf> layers, dmaps;
    TRY(dev_alloc(ctx, L * sizeof(few::LayerPtrs), &layers));
    CK(ctx, cudaMemcpy(layers->p, h.data(), L * sizeof(few::LayerPtrs), cudaMemcpyHostToDevice));
    TRY(dev_alloc(ctx, maps.size() * sizeof(CUtensorMap), &dmaps));
    CK(ctx, cudaMemcpy(dmaps->p, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
    m->few_layers = layers;
    m->few_maps = dmaps;
    return B200NN_OK;
}

int launch_decode_few(b200nn_session *s, int n_steps) {
    b200nn_gpt2 *m = s->gpt2;
    b200nn_ctx *ctx = m->ctx;
    few::Plan p;
    if (!few::make_plan(m, (int)s->batch, (int)s->kv.cap, &p)) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "decode_few: no plan");
    few::Params P = {};
    for (int g = 0; g < few::MATS; ++g) P.mat[g] = p.mat[g];
    P.layers = (const few::LayerPtrs *)m->few_layers->p;
    P.maps = (const CUtensorMap *)m->few_maps->p;
    P.lnf_g = (const float *)m->lnf_g->p;
    P.lnf_b = (const float *)m->lnf_b->p;
    P.wte = (const float *)m->wte->p;
    P.wpe = (const float *)m->wpe->p;
    P.kc = s->kv.kl(0);
    P.vc = s->kv.vl(0);
    P.kv_layer = s->kv.layer_stride();
    P.n_layer = m->cfg.n_layer;
    P.M = (int)s->batch;
    P.d = m->cfg.n_embd;
    P.H = m->cfg.n_head;
    P.cap = (int)s->kv.cap;
    P.vocab = m->cfg.vocab_size;
    P.n_positions = m->cfg.n_positions;
    P.act = m->act();
    P.group_kb = m->int4 ? m->blocks[0].qkv.q.group / 64 : 1;
    P.eps = m->cfg.layer_norm_epsilon;
    P.tok = (uint32_t *)s->ws_step.tok->p;
    P.history = (uint32_t *)s->history->p;
    P.hist_cap = (int)s->hist_cap;
    P.counters = s->pos_ptr();
    P.logits = s->flags & B200NN_TOKENS_ONLY ? nullptr : (float *)s->ws_step.logits->p;
    P.keep_last = s->flags & B200NN_ARGMAX_LAST ? 1 : 0;
    P.words = (uint32_t *)s->few_words->p;
    P.slot_words = (int)p.slot_words;
    P.o_att = (int)p.o_att;
    P.o_lse = (int)p.o_lse;
    P.o_out = (int)p.o_out;
    P.o_fc = (int)p.o_fc;
    P.o_fp = (int)p.o_fp;
    P.state = P.words + p.words;
    P.fenced = P.state + 32; // in a line of its own
    P.dev_err = ctx->dev_err;
    P.wait_cycles = ctx->persist_wait_cycles > 0 ? ctx->persist_wait_cycles : 2000000000LL;
    P.fault_layer = ctx->few_fault_layer;
    P.n_steps = n_steps;
    P.att_splits = p.att_splits;
    P.slots = p.slots;
    P.slot_bytes = p.slot_bytes;
    P.max_parts = p.max_parts;
    P.xs_ld = p.xs_ld;
    void *args[] = {&P};
    CK(ctx, cudaLaunchCooperativeKernel((const void *)few::kernel_of(m->int4, p.MT), dim3(p.grid), dim3(few::THREADS), args, p.smem, ctx->stream));
    CK_LAUNCH(ctx, "decode_few_kernel");
    return B200NN_OK;
}
